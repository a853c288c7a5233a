"""Latent attention of prompt portions on the fifth-generation tensor cores, and of decode steps, against float64: lengths around tiles of
128 rows and 64 keys, around pieces of 16 keys, portions that continue sequences, windows, pages smaller and larger than a tile, and stale numbers behind the context."""

import pytest
import torch

pytestmark = pytest.mark.gpu

STEPS = [([1, 2], [0, 0]), ([8, 1, 9], [0, 63, 64]), ([64, 65], [1, 191]), ([130], [0]), ([3, 40], [500, 0]), ([300, 1, 1], [0, 128, 700])]
DECODE = [([1] * 6, [0, 15, 16, 63, 64, 65]), ([1], [5000]), ([1, 1, 1], [700, 2047, 191])]


@pytest.fixture(autouse=True)
def decode_steps_of_any_size(monkeypatch):
    """(the kernel of decode steps is in use only from the sizes on where it is faster)"""
    from miniserve_b200 import kernels

    monkeypatch.setattr(kernels, "LATENT_DECODE_KEYS", 0)


@pytest.mark.parametrize("rank,rot,heads,page", [(256, 32, 16, 64), (256, 32, 8, 16), (256, 64, 16, 128), (256, 0, 4, 8), (128, 16, 16, 32),
                                                 (64, 48, 1, 64), (64, 64, 128, 64), (128, 32, 32, 192)])
@pytest.mark.parametrize("new,before", STEPS + DECODE)
@pytest.mark.parametrize("window", [None, 70])
def test_against_float64(rank, rot, heads, page, new, before, window):
    from miniserve_b200 import kernels

    g = torch.Generator(device="cuda").manual_seed(rank + heads + sum(new))
    dk, scale, n = rank + rot, (rank + rot) ** -0.5, sum(new)
    assert kernels.library().ms_latent_attention_tcgen05_supports(rank, rot, heads, page)
    lens = [a + b for a, b in zip(new, before)]
    counts = [(length + page - 1) // page for length in lens]
    pages = torch.randperm(sum(counts), generator=g, device="cuda").to(torch.int32)
    cache = torch.full((sum(counts), page, dk), float("nan"), device="cuda").bfloat16()      # (stale rows: nothing of them may be seen)
    tables = torch.zeros((len(new), max(counts) + 1), dtype=torch.int32, device="cuda")
    rows, at = [], 0
    for r, (length, count) in enumerate(zip(lens, counts)):
        tables[r, :count] = pages[at:at + count]
        keys = (torch.randn((length, dk), generator=g, device="cuda") * 1.5).bfloat16()
        keys[length // 2] *= 4                                             # (maxima that grow by more than 2^8 on the way)
        filled = cache[pages[at:at + count].long()].reshape(count * page, dk)
        filled[:length] = keys
        cache[pages[at:at + count].long()] = filled.view(count, page, dk)
        rows.append(keys.double())
        at += count
    q = (torch.randn((n, heads, dk), generator=g, device="cuda") * 2).bfloat16()
    starts = [sum(new[:i]) for i in range(len(new) + 1)]

    def ints(values):
        return torch.tensor(values, dtype=torch.int32, device="cuda")

    positions = ints([p for a, b in zip(new, before) for p in range(b, b + a)])
    requests = ints([r for r, a in enumerate(new) for _ in range(a)])
    out = torch.full((n, heads, rank), float("nan"), device="cuda").bfloat16()
    kernels.latent_attention(q, cache, tables, requests, positions, ints(starts), ints(lens), max(new), max(lens), rank, scale, window, out)
    kernels.check_device_errors(q.device)
    for r, (a, b) in enumerate(zip(new, before)):
        here, keys = q[starts[r]:starts[r + 1]].double(), rows[r]
        scores = torch.einsum("thd,kd->htk", here, keys) * scale
        key, token = torch.arange(a + b, device="cuda")[None, :], (b + torch.arange(a, device="cuda"))[:, None]
        seen = (key <= token) & (key > token - (window or 1 << 30))
        p = torch.softmax(scores.masked_fill(~seen, -torch.inf), dim=-1)
        want = torch.einsum("htk,kd->thd", p, keys[:, :rank])
        # probabilities rounded to bfloat16 (2^-9 of each, in the sum too) and the result once more: 3 2^-9 of the sums of magnitudes; and scores
        # in float32, off by at most dk 2^-23 of the sums of their products' magnitudes, in a probability and in the sum of all
        size = torch.einsum("htk,kd->thd", p, keys[:, :rank].abs())
        products = torch.einsum("thd,kd->htk", here.abs(), keys.abs()) * scale
        slack = 2 * dk * 2.0 ** -23 * (products * seen).amax(dim=-1).T[:, :, None]
        assert float(slack.max()) < 2.0 ** -6
        assert torch.all((out[starts[r]:starts[r + 1]].double() - want).abs() <= (2.0 ** -7 + slack) * size + 1e-6)


def test_contexts_of_one_piece_after_a_step_of_stale_numbers():
    """A warp whose range is one piece of sixteen keys, not all of them real, reads zeros behind the context, whatever the step before (of
    NaN alone) has left in shared memory: a row of ones is then the answer exactly, since all keys have the same score."""
    from miniserve_b200 import kernels

    heads, rank, dk, page, n = 16, 256, 288, 64, 63
    lens = torch.arange(1, n + 1, dtype=torch.int32, device="cuda")
    starts, tables = torch.arange(n + 1, dtype=torch.int32, device="cuda"), torch.arange(n, dtype=torch.int32, device="cuda")[:, None].contiguous()
    zeros = torch.zeros(n, dtype=torch.int32, device="cuda")
    q = torch.ones((n, heads, dk), device="cuda").bfloat16()
    stale = torch.full((n, page, dk), float("nan"), device="cuda").bfloat16()
    cache = stale.clone()
    for r in range(n):
        cache[r, :r + 1] = 1.0
    out = torch.empty((n, heads, rank), device="cuda").bfloat16()
    for _ in range(20):
        for pool in (stale, cache):
            kernels.latent_attention(q, pool, tables, zeros, lens - 1, starts, lens, 1, n, rank, dk ** -0.5, None, out)
        kernels.check_device_errors(q.device)
        assert torch.all(out == 1.0)


@pytest.mark.parametrize("rot,heads,window", [(32, 16, None), (64, 8, None), (32, 20, 2500)])
def test_a_request_is_attended_to_by_what_its_own_keys_ask_for(monkeypatch, rot, heads, window):
    """A captured step knows the longest context allowed, not the step's: which of the two ways a request takes is its own length's choice,
    on the device.  One graph, replayed with short, long and mixed contexts, gives a short request the bits that the way for short
    ones gives alone, and a long one those of the way for long ones."""
    from miniserve_b200 import kernels

    rank, page, limit, n = 256, 64, 40960, 48 if heads == 16 else 64
    dk, border = rank + rot, 98304 // (n * ((heads + 15) // 16))
    assert border <= (window or border)
    g = torch.Generator(device="cuda").manual_seed(heads)
    cache = torch.randn((1 + (2 * border) // page, page, dk), generator=g, device="cuda").bfloat16()       # (all requests see the same pages)
    tables = torch.arange(cache.shape[0], dtype=torch.int32, device="cuda").repeat(n, 1)
    q = torch.randn((n, heads, dk), generator=g, device="cuda").bfloat16()
    starts, zeros = torch.arange(n + 1, dtype=torch.int32, device="cuda"), torch.zeros(n, dtype=torch.int32, device="cuda")
    lens, out = torch.full((n,), 3, dtype=torch.int32, device="cuda"), torch.empty((n, heads, rank), device="cuda").bfloat16()

    def step():
        kernels.latent_attention(q, cache, tables, zeros, lens - 1, starts, lens, 1, limit, rank, dk ** -0.5, window, out)

    found = {}
    for name, keys in (("shared tiles", 1 << 60), ("own pieces", 0), ("rule", 98304)):
        monkeypatch.setattr(kernels, "LATENT_DECODE_KEYS", keys)
        step()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            step()
        for mixture in ([1, border - 1, border, 2 * border], [17, 300], [border + 1, 2 * border - 5]):
            lens.copy_(torch.tensor(mixture * n, dtype=torch.int32)[:n])
            graph.replay()
            found.setdefault(name, []).append((lens.clone(), out.clone()))
    kernels.check_device_errors(q.device)
    for (now, out_tiles), (_, out_pieces), (_, out_rule) in zip(*(found[name] for name in ("shared tiles", "own pieces", "rule"))):
        short = now < border
        assert torch.equal(out_rule[short], out_tiles[short]) and torch.equal(out_rule[~short], out_pieces[~short])
        assert not short.any() or not torch.equal(out_tiles[short], out_pieces[short])


@pytest.mark.parametrize("n,heads,bound,taken", [(2, 16, 49151, False), (2, 16, 49152, True), (3, 16, 40960, True), (3, 16, 32767, False),
                                                 (64, 16, 1536, True), (64, 16, 1535, False), (64, 17, 768, True), (64, 17, 767, False)])
def test_which_decode_steps_may_take_it(monkeypatch, n, heads, bound, taken):
    from miniserve_b200 import kernels

    monkeypatch.setattr(kernels, "LATENT_DECODE_KEYS", 98304)
    lib, calls = kernels.library(), []
    real = lib.ms_latent_decode
    monkeypatch.setattr(lib, "ms_latent_decode", lambda *a: calls.append(1) or real(*a))
    q, cache = torch.ones((n, heads, 288), device="cuda").bfloat16(), torch.ones((1, 64, 288), device="cuda").bfloat16()
    ints = [torch.zeros((n, 1), dtype=torch.int32, device="cuda"), torch.zeros(n, dtype=torch.int32, device="cuda")]
    lens, out = torch.full((n,), 5, dtype=torch.int32, device="cuda"), torch.empty((n, heads, 256), device="cuda").bfloat16()
    kernels.latent_attention(q, cache, ints[0], ints[1], lens - 1, torch.arange(n + 1, dtype=torch.int32, device="cuda"), lens, 1, bound, 256,
                             0.1, None, out)
    assert bool(calls) is taken and torch.all(out == 1.0)


@pytest.mark.parametrize("rank,rot,heads,page", [(256, 32, 16, 64), (256, 64, 8, 16), (128, 32, 16, 32), (64, 16, 4, 128)])
@pytest.mark.parametrize("new", [1, 3])
@pytest.mark.parametrize("window", [None, 70])
def test_the_key_at_a_border_decides(rank, rot, heads, page, new, window):
    """One key's score is far above all others': the first or the last of a piece, a tile, a range, a page or the window, the newest, or one just
    out of sight.  A key too many or too few changes the whole output."""
    from miniserve_b200 import kernels

    dk, g = rank + rot, torch.Generator(device="cuda").manual_seed(rank + heads)
    cases = []
    for length in (16, 17, 64, 65, 129, 400, 1300):
        borders = {0, 15, 16, 31, 32, 63, 64, 127, 128, 191, 192, 255, 256, 639, 640, length - 2, length - 1}
        if window:
            borders |= {length - window - d for d in range(-1, new + 2)} | {(length - window) // 64 * 64}
        cases += [(length, b) for b in sorted(borders) if 0 <= b < length]
    width = (1300 + page - 1) // page
    lens = torch.tensor([length for length, _ in cases], dtype=torch.int32, device="cuda")
    n = len(cases)
    cache = torch.full((n, width * page, dk), float("nan"), device="cuda").bfloat16()
    for r, (length, border) in enumerate(cases):
        cache[r, :length, :rank] = torch.randn((length, rank), generator=g, device="cuda").bfloat16()
        cache[r, :length, rank:] = 0
        cache[r, border, rank] = 16.0
    tables = torch.arange(n * width, dtype=torch.int32, device="cuda").view(n, width)
    q = torch.zeros((n * new, heads, dk), device="cuda").bfloat16()
    q[:, :, rank] = 1.0
    starts = torch.arange(n + 1, dtype=torch.int32, device="cuda") * new
    positions = (lens[:, None] - new + torch.arange(new, device="cuda")).flatten().to(torch.int32)
    requests = torch.arange(n, device="cuda").repeat_interleave(new).to(torch.int32)
    out = torch.empty((n * new, heads, rank), device="cuda").bfloat16()
    kernels.latent_attention(q, cache.view(n * width, page, dk), tables, requests, positions, starts, lens, new, 1300, rank, 1.0, window, out)
    kernels.check_device_errors(q.device)
    for r, (length, border) in enumerate(cases):
        for t in range(new):
            last = length - new + t
            first = max(0, last - window + 1) if window else 0
            rows = cache[r, first:last + 1].double()
            p = torch.softmax(rows[:, rank], dim=0)
            want, size = p @ rows[:, :rank], p @ rows[:, :rank].abs()
            assert torch.all((out[r * new + t].double() - want).abs() <= 2.0 ** -7 * size + 1e-6), (length, border, t)


@pytest.mark.parametrize("new", [1, 80])
def test_the_rounding_of_a_probability_does_not_scale_the_output(new):
    """A key whose score lies 2^2 to 2^7.9 above the first ones' is what most of the output is.  Nothing is rescaled for that, so its probability
    is no power of two, and is rounded: if the sum were that of the unrounded ones, every output would be off by that rounding too. (Measured
    against the result's own rounding to bfloat16; both errors together would be 1.4 times that.)"""
    from miniserve_b200 import kernels

    heads, rank, rot, page, keys, n = 16, 256, 32, 64, 300, 40
    dk, g = rank + rot, torch.Generator(device="cuda").manual_seed(new)
    cache = torch.randn((5, page, dk), generator=g, device="cuda").bfloat16()
    level = torch.full((5 * page,), -20.0, device="cuda")                          # of a key's score, in units of a token's
    level[:160:16], level[210] = 1.0, 2.0                                          # (the first piece of every warp and range has one)
    cache.view(-1, dk)[:, rank:] = 0
    cache.view(-1, dk)[:, rank] = level.bfloat16()
    q = torch.zeros((n * new, heads, dk), device="cuda").bfloat16()
    unit = (2.0 + 5.9 * torch.rand((n * new, heads), generator=g, device="cuda")).bfloat16()     # base-2 distance of the two levels
    q[:, :, rank] = unit
    lens = torch.full((n,), keys, dtype=torch.int32, device="cuda")
    starts = torch.arange(n + 1, dtype=torch.int32, device="cuda") * new
    positions = (torch.arange(new, device="cuda") + keys - new).repeat(n).to(torch.int32)
    requests = torch.arange(n, device="cuda").repeat_interleave(new).to(torch.int32)
    tables = torch.arange(5, dtype=torch.int32, device="cuda").repeat(n, 1)
    scale = 0.6931471805599453
    out = torch.empty((n * new, heads, rank), device="cuda").bfloat16()
    kernels.latent_attention(q, cache, tables, requests, positions, starts, lens, new, keys, rank, scale, None, out)
    kernels.check_device_errors(q.device)
    rows = cache.view(-1, dk)[:keys].double()
    scores = torch.einsum("thd,kd->thk", q.double(), rows) * scale
    scores = scores.masked_fill(torch.arange(keys, device="cuda") > positions[:, None, None], -torch.inf)
    want = torch.einsum("thk,kd->thd", torch.softmax(scores, dim=-1), rows[:, :rank])
    off, rounding = (out.double() - want).norm(), (want.bfloat16().double() - want).norm()
    assert off <= 1.15 * rounding
