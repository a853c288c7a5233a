"""The decode step's fused attention brings whole tiles of keys where they lie within a page and single pieces of sixteen bytes where they do
not: the same cache in pages of any size gives the same bits, whatever lies behind a request's context in its last page."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def in_pages(rows, lengths, page_size, fill):
    """[tokens, heads, d] per request as a pool [pages, heads, page_size, d] with its pages in a shuffled order, and the tables; ``fill`` elsewhere."""
    needed = [(n + page_size - 1) // page_size for n in lengths]
    order = torch.randperm(sum(needed) + 2, generator=torch.Generator().manual_seed(page_size)).tolist()
    heads, d = rows.shape[1:]
    pool = torch.full((len(order), heads, page_size, d), fill, dtype=rows.dtype, device="cuda")
    tables = torch.zeros((len(lengths), max(needed)), dtype=torch.int32)
    at = 0
    for r, n in enumerate(lengths):
        for j in range(needed[r]):
            tables[r, j] = page = order.pop()
            part = rows[at + j * page_size:at + min(n, (j + 1) * page_size)]
            pool[page, :, :part.shape[0]] = part.transpose(0, 1)
        at += n
    return pool, tables.cuda()


@pytest.mark.parametrize("d,n_q,n_kv,window", [(128, 16, 8, None), (128, 9, 3, 70), (64, 8, 2, None), (64, 16, 1, 65)])
@pytest.mark.parametrize("lengths", [[1, 31, 32, 33, 64, 65, 700], [4097], [127, 128, 2111]])
def test_the_page_size_changes_no_bit(lengths, d, n_q, n_kv, window):
    from miniserve_b200 import kernels

    g = torch.Generator().manual_seed(d + len(lengths))
    n, total = len(lengths), sum(lengths)
    rand = lambda *shape: torch.randn(shape, generator=g).to(torch.bfloat16).cuda()
    k_rows, v_rows, qkv = rand(total, n_kv, d), rand(total, n_kv, d), rand(n, (n_q + 2 * n_kv) * d)
    starts = torch.arange(n + 1, dtype=torch.int32, device="cuda")
    lens = torch.tensor(lengths, dtype=torch.int32, device="cuda")
    found = []
    for page_size in (24, 32, 64, 128, 192):
        k_pool, tables = in_pages(k_rows, lengths, page_size, float("nan"))
        v_pool, _ = in_pages(v_rows, lengths, page_size, float("nan"))
        slots = [int(tables[r, (length - 1) // page_size]) * page_size + (length - 1) % page_size for r, length in enumerate(lengths)]
        if n > 2:
            slots[2] = -1                              # (this request's newest key and value are in the cache already)
        out = torch.full((n, n_q, d), 7.0, dtype=torch.bfloat16, device="cuda")
        kernels.decode_attention_fused(qkv, torch.tensor(slots, dtype=torch.int32, device="cuda"), None, None, 1e-6, None, k_pool, v_pool,
                                       tables, starts, lens, max(lengths), d ** -0.5, window, n_q, n_kv, d, out)
        kernels.check_device_errors(out.device)
        found.append(out)
    assert torch.isfinite(found[0].float()).all()
    assert all(torch.equal(found[0], other) for other in found[1:])


@pytest.mark.parametrize("rows,head_dim,group,page_size,want", [
    (2, 128, 2, 16, False), (3, 128, 2, 16, True), (9, 128, 2, 16, False), (1, 128, 2, 32, True), (64, 128, 8, 64, True), (65, 128, 2, 64, False),
    (1, 64, 2, 32, False), (1, 64, 2, 128, True), (2, 128, 9, 64, False), (5, 128, 16, 64, True), (2, 0, 0, 0, False), (8, 0, 0, 0, True)])
def test_which_decode_steps_take_it(rows, head_dim, group, page_size, want):
    from miniserve_b200 import kernels

    assert kernels.decode_attention_fused_preferred(rows, head_dim, group, page_size) is want
