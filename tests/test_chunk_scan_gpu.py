"""The recurrences with a decay per token and head, scanned as matrix products over chunks of 64 tokens: every form against the definition
in float64 and against the walk, token after token, at lengths around the borders of chunks and of the kernels' bands and tiles."""

import pytest
import torch

pytestmark = pytest.mark.gpu

LENGTHS = [[64], [128, 1, 0, 65], [129, 63], [1, 200, 7], [96, 97, 98, 2, 511]]
SIZES = [(4, 2, 128, 128), (2, 2, 64, 64), (3, 3, 40, 56), (2, 1, 100, 130), (1, 1, 33, 3), (2, 2, 128, 259), (2, 1, 6, 17)]


@pytest.fixture(autouse=True)
def in_chunks_from_96_tokens_on(monkeypatch):
    """(in use only from the sizes on where it is faster)"""
    from miniserve_b200 import kernels

    for name, value in (("CHUNK_SCAN_LONGEST", 0), ("CHUNK_SCAN_DELTA", 0)):
        monkeypatch.setattr(kernels, name, value)
    lib, scans = kernels.library(), []
    for name in ("ms_chunk_scan", "ms_selective_chunk_scan"):
        monkeypatch.setattr(lib, name, lambda *args, real=getattr(lib, name): scans.append(1) or real(*args))
    yield
    assert len(scans) >= 1                             # (not the walk compared with itself)


def ints(values):
    return torch.tensor(values, dtype=torch.int32, device="cuda")


def recurrence(form, q, k, v, keep, write, state):
    """All heads in float64: q, k [T, H, dim], v [T, H, vdim], keep, write [T, H]; rows of y [T, H, columns] (memory: the read-outs of n
    last), the state [H, columns, dim] afterwards."""
    s, rows = state.clone(), []
    if form == "memory":
        v = torch.cat([v, torch.ones_like(v[:, :, :1])], dim=2)
    for t in range(q.shape[0]):
        s = keep[t, :, None, None] * s
        seen = (s @ k[t, :, :, None])[:, :, 0] if form == "delta" else 0
        s = s + (write[t, :, None] * (v[t] - seen))[:, :, None] * k[t, :, None, :]
        rows.append((s @ q[t, :, :, None])[:, :, 0])
    return torch.stack(rows) if rows else v[:, :, :1].expand(0, s.shape[0], s.shape[1]), s


def problem(form, dtype, lengths, heads, kv_heads, dim, vdim, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    n, columns = sum(lengths), vdim + 1 if form == "memory" else vdim
    kv_heads = heads if form == "memory" else kv_heads
    pad = 8 if dim % 8 == 0 and vdim % 8 == 0 else 3          # (rows on 16-byte boundaries, or not)
    rows = (torch.randn((n, 2 * kv_heads * dim + heads * vdim + pad), generator=g, device="cuda") * 0.5)
    q_col, k_col, v_col = 0, kv_heads * dim, 2 * kv_heads * dim
    if form == "delta":
        keys = rows[:, k_col:v_col].view(n, kv_heads, dim)
        rows[:, k_col:v_col] = (keys / keys.norm(dim=-1, keepdim=True)).reshape(n, -1)
    rows = rows.to(dtype)
    uniform = torch.rand((n, heads, 3), generator=g, device="cuda")
    gates = uniform.clone()
    gates[:, :, 0] = torch.where(uniform[:, :, 1] < 0.1, uniform[:, :, 0] * 0.5, 0.9 + 0.1 * uniform[:, :, 0])     # some forget much
    gates = gates[:, :, :3 if form == "memory" else 2].contiguous()
    if form == "decay":
        gates = 0.5 + 0.5 * torch.rand((heads,), generator=g, device="cuda")
    slots = torch.randperm(len(lengths) + 1, generator=g, device="cuda")[:len(lengths)]
    states = torch.randn((len(lengths) + 1, 5 + heads * columns * dim + 2), generator=g, device="cuda") * 0.3
    return rows, (q_col, k_col, v_col), gates, slots, states, kv_heads, columns


def run(form, rows, cols, gates, slots, states, lengths, heads, kv_heads, dim, vdim, scale=0.7, **options):
    from miniserve_b200 import kernels

    n = rows.shape[0]
    y = torch.full((n, heads, vdim), float("nan"), device="cuda")
    bottom = torch.full((n, heads), float("nan"), device="cuda") if form == "memory" else None
    starts = [0]
    for length in lengths:
        starts.append(starts[-1] + length)
    kernels.matrix_scan(form, rows, cols[0], rows, cols[1], rows, cols[2], gates, states, 5, slots.to(torch.int32), ints(starts), max(lengths),
                        heads, kv_heads, dim, vdim, y, q_scale=scale, bottom=bottom, **options)
    return y, bottom


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("form", ["memory", "delta", "decay"])
@pytest.mark.parametrize("heads,kv_heads,dim,vdim", SIZES)
@pytest.mark.parametrize("lengths", LENGTHS)
def test_matrix_scan_in_chunks(form, dtype, heads, kv_heads, dim, vdim, lengths):
    from miniserve_b200 import kernels

    if max(lengths) < 96:
        lengths = lengths + [96]                       # (shorter steps are walked)
    rows, cols, gates, slots, states, kv_heads, columns = problem(form, dtype, lengths, heads, kv_heads, dim, vdim, 5 + dim + vdim)
    assert kernels.library().ms_chunk_scan_chunk(len(lengths), max(lengths), heads, dim) == 64
    options = dict(input_activation="silu") if form == "decay" else {}
    start, walked = states.clone(), states.clone()
    y, bottom = run(form, rows, cols, gates, slots, states, lengths, heads, kv_heads, dim, vdim, **options)
    y_walk, bottom_walk = run(form, rows, cols, gates, slots, walked, lengths, heads, kv_heads, dim, vdim, chunk=0, **options)
    at, off, off_walk = 0, 0.0, 0.0
    for r, length in enumerate(lengths):
        here = rows[at:at + length].double()
        if form == "decay":
            here = here * torch.sigmoid(here)
        q, k = (here[:, c:c + kv_heads * dim].view(length, kv_heads, dim).repeat_interleave(heads // kv_heads, 1) for c in cols[:2])
        v = here[:, cols[2]:cols[2] + heads * vdim].view(length, heads, vdim)
        here_gates = gates[at:at + length].double() if form != "decay" else None
        keep = gates.double().expand(length, heads) if form == "decay" else here_gates[:, :, 0]
        write = torch.ones_like(keep) if form == "decay" else here_gates[:, :, 1]
        span = slice(5, 5 + heads * columns * dim)
        want, after = recurrence(form, 0.7 * q, k, v, keep, write, start[slots[r], span].double().view(heads, columns, dim))
        for found, reads, state, walk in ((y, bottom, states, False), (y_walk, bottom_walk, walked, True)):
            errors = [found[at:at + length].double() - want[:, :, :vdim], state[slots[r], span].double() - after.flatten()]
            if form == "memory":
                errors.append(reads[at:at + length].double() - (torch.maximum(want[:, :, vdim].abs(), here_gates[:, :, 2]) + 1e-6))
            worst = max(float(e.abs().max()) if e.numel() else 0.0 for e in errors)
            off, off_walk = (off, max(off_walk, worst)) if walk else (max(off, worst), off_walk)
        at += length
    scale = max(1.0, float(y_walk.abs().max()))
    assert off <= 2e-5 * scale                              # the walk's own bound
    assert off <= 3 * off_walk + 1e-6 * scale               # and no less exact than the walk (maxima of few thousand roundings)
    untouched = torch.ones(states.shape[0], dtype=torch.bool, device="cuda")
    untouched[slots[[i for i, length in enumerate(lengths) if length]]] = False
    assert torch.equal(states[untouched], start[untouched]) and torch.equal(states[:, :5], start[:, :5]) and torch.equal(states[:, -2:], start[:, -2:])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("form", ["memory", "delta", "decay"])
@pytest.mark.parametrize("heads,kv_heads,dim,vdim", [(20, 5, 128, 136), (21, 7, 40, 130), (16, 16, 64, 64)])
def test_a_block_reads_several_tiles_heads_chunks_and_requests(form, dtype, heads, kv_heads, dim, vdim):
    """More than two blocks a multiprocessor have work for, of more requests than a warp has lanes, some without tokens: the walk's rows.
    (Either way is within 2e-5 of the definition, see above: 4e-5 apart.)"""
    lengths = [1, 0, 65, 3, 130] * 7 + [0, 0, 200, 64]
    rows, cols, gates, slots, states, kv_heads, columns = problem(form, dtype, lengths, heads, kv_heads, dim, vdim, 11 + dim)
    options = dict(input_activation="silu") if form == "decay" else {}
    walked = states.clone()
    y, bottom = run(form, rows, cols, gates, slots, states, lengths, heads, kv_heads, dim, vdim, **options)
    y_walk, bottom_walk = run(form, rows, cols, gates, slots, walked, lengths, heads, kv_heads, dim, vdim, chunk=0, **options)
    pairs = [(y, y_walk), (states, walked)] + ([(bottom, bottom_walk)] if form == "memory" else [])
    scale = max(1.0, float(y_walk.abs().max()))
    assert all(float((a.double() - b.double()).abs().max()) <= 4e-5 * scale for a, b in pairs)


@pytest.mark.parametrize("heads,P,N,G", [(4, 64, 128, 2), (3, 64, 64, 1), (2, 40, 24, 2), (2, 130, 100, 1), (1, 3, 7, 1)])
@pytest.mark.parametrize("lengths", LENGTHS)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_selective_scan_in_chunks(dtype, heads, P, N, G, lengths):
    from miniserve_b200 import kernels

    if max(lengths) < 96:
        lengths = lengths + [96]
    g = torch.Generator(device="cuda").manual_seed(3 + P + N)
    n, inner = sum(lengths), heads * P
    conv = torch.randn((n, inner + 2 * G * N), generator=g, device="cuda") * 0.5
    proj = (torch.randn((n, heads + 2), generator=g, device="cuda") * 2).to(dtype)
    dt_bias, a_log, skip = (torch.randn(heads, generator=g, device="cuda") for _ in range(3))
    slots = torch.randperm(len(lengths) + 1, generator=g, device="cuda")[:len(lengths)]
    start = torch.randn((len(lengths) + 1, 3 + inner * N), generator=g, device="cuda") * 0.3
    starts = [0]
    for length in lengths:
        starts.append(starts[-1] + length)
    found = []
    for chunked in (True, False):
        states, y = start.clone(), torch.full((n, inner), float("nan"), device="cuda")
        kernels.selective_scan(conv, proj, 1, dt_bias, a_log, skip, states, 3, slots.to(torch.int32), ints(starts), heads, P, N, G, y,
                               max_query_len=max(lengths), chunked=chunked)
        found.append((y, states))
    off = [0.0, 0.0]
    for r, length in enumerate(lengths):
        here = conv[starts[r]:starts[r + 1]].double()
        if not length:
            continue
        b, c = (here[:, at:at + G * N].view(length, G, N).repeat_interleave(heads // G, 1) for at in (inner, inner + G * N))
        x = here[:, :inner].view(length, heads, P)
        dt = torch.nn.functional.softplus(proj[starts[r]:starts[r + 1], 1:1 + heads].double() + dt_bias.double())
        want, after = recurrence("ssm", c, b, x, torch.exp(-torch.exp(a_log.double()) * dt), dt, start[slots[r], 3:].double().view(heads, P, N))
        want = (want + skip.double()[:, None] * x).reshape(length, inner)
        for i, (y, states) in enumerate(found):
            off[i] = max(off[i], float((y[starts[r]:starts[r + 1]].double() - want).abs().max()),
                         float((states[slots[r], 3:].double() - after.flatten()).abs().max()))
    scale = max(1.0, float(found[1][0].abs().max()))
    assert off[0] <= 2e-5 * scale and off[0] <= 3 * off[1] + 1e-6 * scale
    assert torch.equal(found[0][1][:, :3], start[:, :3])


@pytest.mark.parametrize("form", ["memory", "delta", "decay"])
def test_an_infinity_reaches_no_token_before_it(form):
    """A chunk's products run over all its tokens at once; what a token must not see is left out, not multiplied by zero."""
    lengths, bad = [150], 101
    rows, cols, gates, slots, states, kv_heads, columns = problem(form, torch.float32, lengths, 2, 2, 64, 64, 9)
    clean, _ = run(form, rows, cols, gates, slots, states.clone(), lengths, 2, kv_heads, 64, 64)
    rows[bad] = float("inf")
    y, _ = run(form, rows, cols, gates, slots, states, lengths, 2, kv_heads, 64, 64)
    assert torch.equal(y[:bad], clean[:bad]) and not torch.isfinite(y[bad:]).all()
