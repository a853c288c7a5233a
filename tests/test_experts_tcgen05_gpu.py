"""The experts' products on the fifth-generation tensor cores, against float64: segments that are empty, of one row, around a tile of 128
and of several tiles, remainders in columns and inner size, every activation, rows gathered and in place."""

import pytest
import torch

pytestmark = pytest.mark.gpu

SEGMENTS = [[1], [0, 1, 0, 3], [128, 127, 129, 0], [5] * 40, [300, 0, 17, 256, 1], [513, 2]]


@pytest.mark.parametrize("n,k", [(8, 8), (128, 64), (136, 72), (256, 200), (520, 1408), (2816, 136)])
@pytest.mark.parametrize("segments", SEGMENTS)
@pytest.mark.parametrize("activation", ["none", "relu_square", "clamped_glu", "silu_glu"])
def test_expert_linear(activation, segments, n, k):
    from miniserve_b200 import kernels

    g = torch.Generator(device="cuda").manual_seed(n + k + len(segments))
    experts, pairs, top, limit = len(segments), sum(segments), 2, 1.5
    gated = activation in ("clamped_glu", "silu_glu")
    weight = (torch.randn((experts, n, k), generator=g, device="cuda") * k ** -0.5).bfloat16()
    offsets = torch.tensor([sum(segments[:e]) for e in range(experts + 1)] + [pairs + 3], dtype=torch.int32, device="cuda")   # (one more segment: not computed)
    assert kernels.library().ms_expert_tcgen05_supports(experts, n, k)
    for gathered in (True, False):
        tokens = (pairs + top - 1) // top
        x = torch.randn((tokens if gathered else pairs, k), generator=g, device="cuda").bfloat16()
        order = torch.randperm(tokens * top, generator=g, device="cuda")[:pairs].to(torch.int32) if gathered else None
        scale = torch.rand((pairs if not gathered else tokens * top,), generator=g, device="cuda") + 0.5
        scaled = gathered and activation == "silu_glu" and tokens * top == pairs
        out = torch.full((pairs, n // 2 if gated else n), float("nan"), device="cuda").bfloat16()
        kernels.expert_linear(x, order, top, weight, out, offsets, activation=activation, limit=limit, pair_scale=scale if scaled else None)
        kernels.check_device_errors(x.device)
        rows = x.double()[order.long() // top] if gathered else x.double()
        expert = torch.repeat_interleave(torch.arange(experts, device="cuda"), torch.tensor(segments, device="cuda"))
        want, size = torch.empty((pairs, n), dtype=torch.float64, device="cuda"), torch.empty((pairs, n), dtype=torch.float64, device="cuda")
        for e in range(experts):
            here = expert == e
            want[here], size[here] = rows[here] @ weight[e].double().T, rows[here].abs() @ weight[e].double().abs().T
        # sums of k products in float32, off by at most k 2^-23 of the sum of their magnitudes (an accumulator may truncate), then one
        # rounding to bfloat16
        error = k * 2.0 ** -23 * size
        if activation == "relu_square":
            want = want.clamp(min=0)
            want, error = want ** 2, 2 * want * error + error ** 2
        elif gated:
            gate, up, e_gate, e_up = want[:, 0::2], want[:, 1::2], error[:, 0::2], error[:, 1::2]
            if activation == "clamped_glu":
                gate, up, alpha, plus = gate.clamp(max=limit), up.clamp(-limit, limit), 1.702, 1.0
            else:
                s = scale.double()[order.long()][:, None] if scaled else 1.0
                gate, up, e_gate, e_up, alpha, plus = s * gate, s * up, s * e_gate, s * e_up, 1.0, 0.0
            part = gate * torch.sigmoid(alpha * gate)
            # |d part / d gate| <= 1.1; expf and the division are good to a few 2^-23
            want, error = part * (up + plus), 1.1 * e_gate * (up + plus).abs() + (part.abs() + 1.1 * e_gate) * e_up + 1e-6 * (part * (up + plus)).abs()
        assert torch.all((out.double() - want).abs() <= error + 2.0 ** -8 * (want.abs() + error) + 1e-30)
