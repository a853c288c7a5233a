"""The forms with wide accesses of the kernels around the recurrences and the experts, against the plain operations, at sizes around
their tiles, and against the forms that take any size."""

import pytest
import torch

import plain_ops

pytestmark = pytest.mark.gpu
DTYPES = [torch.bfloat16, torch.float32]


def rand(shape, dtype, seed, std=1.0):
    return (torch.randn(shape, generator=torch.Generator().manual_seed(seed)) * std).to(dtype).cuda()


def ints(values):
    return torch.tensor(values, dtype=torch.int32, device="cuda")


def starts_of(lengths):
    return [sum(lengths[:i]) for i in range(len(lengths) + 1)]


def close(got, want, dtype=torch.float32):
    """A few float32 roundings of the largest; a sum near the middle of two bfloat16 numbers may become either, and neighbours lie up to
    2^-7 of their size apart."""
    scale = float(want.double().abs().max())
    return torch.allclose(got.double().cpu(), want.double().cpu(), atol=2e-5 * scale, rtol=2.0 ** -7 if dtype == torch.bfloat16 else 2e-5)


@pytest.mark.parametrize("heads", [1, 8, 33])
@pytest.mark.parametrize("lengths", [[96], [2047, 1, 0, 9], [2048, 5], [2049], [5000, 97]])
def test_exponential_gates_of_long_portions(heads, lengths):
    """The scan over tokens against the definition in float64: what the factors stand for, whatever maxima stabilise them, are the
    products of forget gates and the input gates; and the maxima themselves."""
    from miniserve_b200 import kernels

    n, cap = sum(lengths), 15.0
    logits = rand((n, 2 * heads), torch.float32, heads, 3.0)
    logits[:, heads:] += 3.0
    states = rand((len(lengths) + 1, heads + 5), torch.float32, 2).abs()
    start, starts, slots = states.clone(), starts_of(lengths), list(range(len(lengths), 0, -1))
    gates = torch.full((n, heads, 3), float("nan"), device="cuda")
    kernels.exponential_gates(logits, cap, states, 2, ints(slots), ints(starts), max(lengths), gates)
    x = logits.double()
    i, f = cap * torch.tanh(x[:, :heads] / cap), torch.nn.functional.logsigmoid(cap * torch.tanh(x[:, heads:] / cap))
    for r, length in enumerate(lengths):
        m = start[slots[r], 2:2 + heads].double()
        for t in range(starts[r], starts[r + 1]):
            before, m = m, torch.maximum(f[t] + m, i[t])
            want = torch.stack([torch.exp(f[t] + before - m), torch.exp(i[t] - m), torch.exp(-m)], dim=-1)
            # maxima of up to 15 in float32, sums of a few dozen roundings: exponents off by some 1e-5
            if t % 61 == 0 or t == starts[r + 1] - 1:
                assert torch.allclose(gates[t].double(), want, rtol=5e-5, atol=1e-30)
        assert torch.allclose(states[slots[r], 2:2 + heads].double(), m, atol=2e-5)
    assert torch.equal(states[0], start[0]) and torch.equal(states[:, :2], start[:, :2]) and torch.equal(states[:, 2 + heads:], start[:, 2 + heads:])


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("divide", [True, False])
@pytest.mark.parametrize("n,heads,vdim", [(1, 1, 4), (3, 3, 128), (7, 5, 132), (5, 2, 256), (2, 3, 260), (9, 1, 512), (33, 16, 64), (2, 2, 516)])
def test_head_norm_gate(dtype, divide, n, heads, vdim):
    from miniserve_b200 import kernels

    y, weight, gate = rand((n, heads, vdim), torch.float32, 1, 3.0), rand((vdim,), torch.float32, 2), rand((n, heads * vdim + 8), dtype, 3, 2.0)
    bottom = (0.1 + rand((n, heads), torch.float32, 4).abs()) if divide else None
    out, want = torch.zeros((n, heads * vdim), dtype=dtype).cuda(), torch.zeros((n, heads * vdim), dtype=dtype)
    for activation in ("sigmoid", "silu"):
        kernels.head_norm_gate(y, bottom, weight, gate, 8, activation, 1e-5, out)
        plain_ops.head_norm_gate(y.cpu(), None if bottom is None else bottom.cpu(), weight.cpu(), gate.cpu(), 8, activation, 1e-5, want)
        assert close(out, want, dtype)


@pytest.mark.parametrize("n,heads,dim,col", [(1, 1, 4, 0), (5, 3, 128, 8), (17, 1, 64, 4), (3, 7, 36, 0), (2, 2, 132, 0)])
def test_unit_norm_heads(n, heads, dim, col):
    from miniserve_b200 import kernels

    x = rand((n, col + heads * dim + 4), torch.float32, 5, 2.0)
    x[0, col:col + dim] = 0.0
    want = x.cpu()
    plain_ops.unit_norm_heads(want, col, heads, dim, 1e-6, 0.3)
    kernels.unit_norm_heads(x, col, heads, dim, 1e-6, 0.3)
    assert close(x, want)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("like_proj", [True, False])
@pytest.mark.parametrize("channels,taps", [(4, 4), (512, 2), (516, 3), (1028, 4)])
def test_convolution(dtype, like_proj, channels, taps):
    """Portions shorter than the taps, as long as a thread's stretch of tokens, and around four tokens at a time."""
    from miniserve_b200 import kernels

    lengths, slots, col = [1, 2, 3, 16, 17, 31, 0, 64], [7, 0, 2, 1, 4, 3, 6, 5], 4
    n = sum(lengths)
    proj, weight = rand((n, col + channels + 4), dtype, 6), rand((channels, taps), torch.float32, 7)
    bias, in_bias = rand((channels,), torch.float32, 8), rand((channels,), torch.float32, 9)
    states = rand((9, 3 + (taps - 1) * channels), torch.float32, 10)
    kind = dtype if like_proj else torch.float32
    out, want, want_states = torch.zeros((n, channels), dtype=kind).cuda(), torch.zeros((n, channels), dtype=kind), states.cpu()
    plain_ops.causal_conv(proj.cpu(), col, weight.cpu(), bias.cpu(), want_states, 3, torch.tensor(slots), torch.tensor(starts_of(lengths)), max(lengths),
                          want, activation="silu", in_bias=in_bias.cpu())
    kernels.causal_conv(proj, col, weight, bias, states, 3, ints(slots), ints(starts_of(lengths)), max(lengths), out, activation="silu", in_bias=in_bias)
    assert close(out, want, kind) and close(states, want_states)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("n,rows,width", [(1, 1, 4), (9, 17, 1024), (8, 8, 1028), (3, 5, 2048), (1030, 16, 132), (65, 70, 3000)])
def test_few_rows_in_float32(dtype, n, rows, width):
    from miniserve_b200 import kernels

    x, weight, bias = rand((n, width), dtype, 11), rand((rows, width), torch.float32, 12), rand((rows,), torch.float32, 13)
    out = torch.full((n, rows), float("nan"), device="cuda")
    kernels.small_linear_f32(x, weight, bias, out)
    want = x.double() @ weight.double().T + bias.double()
    assert torch.all((out.double() - want).abs() <= width * 2.0 ** -24 * (x.double().abs() @ weight.double().abs().T + bias.double().abs()))
    alone = torch.empty((1, rows), device="cuda")
    kernels.small_linear_f32(x[n // 2:n // 2 + 1].contiguous(), weight, bias, alone)
    assert torch.equal(alone[0], out[n // 2])


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("identity", [0, 2])
@pytest.mark.parametrize("n,top,width,weighted,shared", [(1, 1, 8, True, False), (5, 4, 1024, True, True), (3, 5, 1032, False, False), (9, 9, 2048, True, True),
                                                         (4, 3, 36, True, True)])
def test_expert_combine(dtype, identity, n, top, width, weighted, shared):
    from miniserve_b200 import kernels

    if identity and not weighted:
        pytest.skip("identity experts go with weights")
    y, x, own = rand((n * top, width), dtype, 14), rand((n, width), dtype, 15), rand((n, width), dtype, 16)
    place = torch.randperm(n * top, generator=torch.Generator().manual_seed(17)).to(torch.int32).cuda()
    ids = torch.randint(0, 6, (n, top), generator=torch.Generator().manual_seed(18)).to(torch.int32).cuda()
    weights, gate = rand((n, top), torch.float32, 19).abs(), rand((n, 3), torch.float32, 20)
    out = torch.zeros((n, width), dtype=dtype).cuda()
    options = dict(shared_gate=gate, shared_gate_col=1) if shared else {}
    kernels.expert_combine(y, place, weights if weighted else None, own if shared else None, out, ids=ids if identity else None,
                           first_identity=6 - identity, x=x if identity else None, **options)
    rows = y.double()[place.long()].view(n, top, width)
    if identity:
        rows = torch.where((ids >= 6 - identity)[:, :, None], x.double()[:, None, :], rows)
    want = (rows * (weights.double() if weighted else torch.ones_like(weights.double()))[:, :, None]).sum(1)
    if shared:
        want = want + torch.sigmoid(gate[:, 1:2].double()) * own.double()
    assert close(out, want, dtype)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("heads,dim,rot,rank", [(1, 8, 16, 8), (16, 64, 32, 256), (3, 16, 64, 264), (8, 8, 48, 1024)])
def test_latent_prepare_and_head_gate(dtype, heads, dim, rot, rank):
    from miniserve_b200 import kernels

    n = 7
    proj = rand((n, heads * (dim + rot) + rank + rot + 8), dtype, 21)
    slots, weight = ints([3, 0, -1, 9, 5, 6, 1]), rand((rank,), dtype, 22)
    table = rand((n, rot // 2, 2), torch.float32, 23)
    cache, q = rand((10, rank + rot), dtype, 24), rand((n, heads, rank + rot), dtype, 25)
    want_cache, want_q = cache.cpu(), q.cpu()
    args = (0, heads * (dim + rot), heads, dim, rot, rank)
    plain_ops.latent_prepare(proj.cpu(), *args, slots.cpu(), weight.cpu(), 1e-5, table.cpu(), rot, want_cache, want_q)
    kernels.latent_prepare(proj, *args, slots, weight, 1e-5, table, rot, cache.view(1, 10, rank + rot), q)
    assert close(cache, want_cache, dtype) and close(q, want_q, dtype)
    x, gate = rand((n, heads, dim), dtype, 26), rand((n, heads + 3), dtype, 27, 2.0)
    want = x.double() * torch.sigmoid(gate[:, 2:2 + heads].double())[:, :, None]
    kernels.head_gate(x, gate, 2)
    assert close(x, want, dtype)
