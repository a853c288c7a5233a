"""The float32 product on the tensor cores (three bfloat16 parts of each operand) against float64, at sizes around its tiles of rows,
its stages of 64 k and its clusters."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def operands(m, n, k, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(m, k, generator=g, device="cuda"), torch.randn(n, k, generator=g, device="cuda")


@pytest.mark.parametrize("m,n,k", [(1, 1, 1536), (1, 2048, 6144), (16, 128, 1540), (17, 129, 2052), (145, 300, 1604), (144, 4096, 2048), (289, 5000, 1536),
                                   (33, 12288, 1600), (130, 8192, 1024), (700, 2816, 1568), (5, 20000, 1600)])
def test_long_sums(m, n, k):
    """An addition to a stage's sum drops what lies behind 24 bits (up to 2^-23 of what is summed so far, in a stage's last four steps and
    the small products before them), stages are added with one rounding each: (K / 64 + 8) 2^-23 of the sum of the magnitudes is well
    above both.  And a row's bits do not depend on the rows beside it."""
    from miniserve_b200 import kernels

    assert kernels._asked("ms_gemm_f32_tcgen05_takes", n, k)
    x, w = operands(m, n, k, m + n + k)
    out = torch.full((m, n), float("nan"), device="cuda")
    kernels.linear(x, w, out)
    want = x.double() @ w.double().T
    bound = (k / 64 + 8) * 2.0 ** -23 * (x.double().abs() @ w.double().abs().T)
    assert torch.all((out.double() - want).abs() <= bound)
    # the distance that float32 sums in ascending order have grows with sqrt(K / 2) roundings of 2^-25 each; this one must not exceed it
    assert float((out.double() - want).norm() / want.norm()) <= (k / 2) ** 0.5 * 2.0 ** -25
    for row in {0, m // 2, m - 1}:
        alone = torch.empty((1, n), device="cuda")
        kernels.linear(x[row:row + 1].contiguous(), w, alone)
        assert torch.equal(alone[0], out[row])
    kernels.check_device_errors(x.device)


@pytest.mark.parametrize("m,n,k", [(16384, 130, 1536), (16385, 130, 1536), (32768 + 37, 5, 1536), ((1 << 33) // 1536 + 1, 1, 1536)])
def test_many_rows(m, n, k):
    """More rows than are multiplied at a time, and more numbers than 2^33: a row's bits are those that it has alone."""
    from miniserve_b200 import kernels

    x, w = torch.zeros((m, k), device="cuda"), operands(1, n, k, 4)[1]
    looked_at = sorted({0, 1, 16383, m // 2, m - 2, m - 1})
    x[looked_at] = torch.randn((len(looked_at), k), device="cuda")
    out, few = torch.full((m, n), float("nan"), device="cuda"), torch.empty((len(looked_at), n), device="cuda")
    kernels.linear(x, w, out)
    kernels.linear(x[looked_at].contiguous(), w, few)
    assert torch.equal(out[looked_at], few) and torch.count_nonzero(out) == torch.count_nonzero(few) and few.any()
    kernels.check_device_errors(x.device)


def test_scratch_is_bounded():
    from miniserve_b200 import kernels

    assert kernels._asked("ms_gemm_f32_tcgen05_scratch", 1 << 24, 10944) == 6 * 16384 * 10944


@pytest.mark.parametrize("n", [300, 20000])
def test_numbers_at_the_ends_of_the_range(n):
    """Infinities, NaNs, overflowing sums and operands near the largest number give what the plain product gives (one block a tile, and
    clusters)."""
    from miniserve_b200 import kernels

    x, w = operands(37, n, 1600, 3)
    x[3, 5], x[4, 7], w[7, 9], w[n - 1, 1599] = float("inf"), float("nan"), float("-inf"), float("inf")
    x[8], w[11], x[9, 3], w[:, 3] = 3.0e38, 3.0e38, 3.4028e38, 0.25
    out = torch.empty((37, n), device="cuda")
    kernels.linear(x, w, out)
    # the same rows one number past a 16-byte boundary: the plain kernel
    room = torch.empty(37 * 1600 + 1, device="cuda")[1:]
    plain = torch.empty((37, n), device="cuda")
    kernels.linear(room.copy_(x.reshape(-1)).view(37, 1600), w, plain)
    finite = torch.isfinite(plain)
    assert torch.equal(torch.isfinite(out), finite) and not finite[3].any() and torch.isfinite(out[9, :7]).all()
    assert torch.equal(torch.nan_to_num(out, nan=7.0)[~finite], torch.nan_to_num(plain, nan=7.0)[~finite])
    scale = x.double().abs() @ w.double().abs().T
    assert torch.all(((out.double() - plain.double()).abs() <= 1600 * 2.0 ** -23 * scale)[finite])
    kernels.check_device_errors(x.device)


@pytest.mark.parametrize("n", [300, 20000])
@pytest.mark.parametrize("of_x,of_w", [(1e-36, 1.0), (1.0, 1e-36), (1e-18, 1e-18), (3e-34, 0.02)])
def test_small_numbers(n, of_x, of_w):
    """Operands whose parts end before they do (below 2^-110) count whole: the distance that float32 sums have, see above.  Rows of ordinary numbers
    beside them, and zeros, are what they are alone."""
    from miniserve_b200 import kernels

    x, w = operands(21, n, 1600, 9)
    ordinary = torch.empty((21, n), device="cuda")
    kernels.linear(x, w, ordinary)
    x[5:] *= of_x
    x[20] = 0.0
    w[:n - 7] *= of_w
    out = torch.empty((21, n), device="cuda")
    kernels.linear(x, w, out)
    small, want = out[5:20, :n - 7].double(), x[5:20].double() @ w[:n - 7].double().T
    assert float((small - want).norm() / want.norm()) <= 800 ** 0.5 * 2.0 ** -25
    assert torch.equal(out[:5, n - 7:], ordinary[:5, n - 7:]) and not out[20].any()
    kernels.check_device_errors(x.device)


def test_numbers_that_are_not_finite_cost_no_orders_of_magnitude():
    """Sums that are not finite are formed again by whole blocks.  (Measured: all of them 17 times the time of none;
    by a thread for each, 310 times.)"""
    from miniserve_b200 import kernels

    x, w = operands(389, 2048, 6144, 5)
    out, times = torch.empty((389, 2048), device="cuda"), []
    for value in (0.0, float("nan")):
        x[:, 7] = value
        for _ in range(3):
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            start.record()
            kernels.linear(x, w, out)
            end.record()
            end.synchronize()
        times.append(start.elapsed_time(end))
    assert out.isnan().all() and times[1] <= 30 * times[0]
