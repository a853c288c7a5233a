"""The scans in chunks on the tensor cores (chunks of 128 tokens, operands in exact bfloat16 parts): the tests of the scans in chunks at lengths and
sizes around the borders of chunks, tiles of 64 value columns and blocks of 64 key entries, and what only these kernels have."""

import pytest
import torch

import test_chunk_scan_gpu as scans

pytestmark = pytest.mark.gpu

LENGTHS = [[128], [127, 1, 0, 129], [257, 63], [1, 200, 7], [96, 64, 65, 2, 511]]
SIZES = [(4, 2, 128, 128), (2, 2, 64, 64), (3, 3, 40, 56), (2, 1, 100, 130), (1, 1, 33, 3), (2, 2, 128, 259), (2, 1, 6, 17), (2, 1, 72, 64)]


@pytest.fixture
def on_tensor_cores(monkeypatch):
    from miniserve_b200 import kernels

    for name in ("CHUNK_SCAN_LONGEST", "CHUNK_SCAN_DELTA"):
        monkeypatch.setattr(kernels, name, 0)
    monkeypatch.setattr(kernels, "_scanned_on_tensor_cores", lambda *args: True)
    lib, records = kernels.library(), []
    for name in ("ms_chunk_scan", "ms_selective_chunk_scan"):
        monkeypatch.setattr(lib, name, lambda *args, real=getattr(lib, name): records.append(args[-3]) or real(*args))
    yield
    assert records and all(records)                    # (not the float32 pipe)
    kernels.check_device_errors(torch.device("cuda:0"))


@pytest.mark.usefixtures("on_tensor_cores")
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("form", ["memory", "delta"])
@pytest.mark.parametrize("heads,kv_heads,dim,vdim", SIZES)
@pytest.mark.parametrize("lengths", LENGTHS)
def test_against_the_definition(form, dtype, heads, kv_heads, dim, vdim, lengths):
    scans.test_matrix_scan_in_chunks(form, dtype, heads, kv_heads, dim, vdim, lengths)


@pytest.mark.usefixtures("on_tensor_cores")
@pytest.mark.parametrize("heads,P,N,G", [(4, 64, 128, 2), (3, 64, 64, 1), (2, 40, 24, 2), (2, 130, 100, 1), (1, 3, 7, 1)])
@pytest.mark.parametrize("lengths", LENGTHS)
def test_selective(heads, P, N, G, lengths):
    scans.test_selective_scan_in_chunks(torch.bfloat16, heads, P, N, G, lengths)


@pytest.mark.usefixtures("on_tensor_cores")
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("form", ["memory", "delta", "decay"])
@pytest.mark.parametrize("heads,kv_heads,dim,vdim", [(20, 5, 128, 136), (21, 7, 40, 130), (16, 16, 64, 64)])
def test_runs_of_units(form, dtype, heads, kv_heads, dim, vdim):
    """More units than multiprocessors, of more requests than a warp has lanes, some without tokens, some too short: the walk's rows.  (Either
    way is within 2e-5 of the definition, see there: 4e-5 apart.)"""
    lengths = [1, 0, 65, 3, 130] * 7 + [0, 0, 200, 64]
    rows, cols, gates, slots, states, kv_heads, columns = scans.problem(form, dtype, lengths, heads, kv_heads, dim, vdim, 11 + dim)
    walked = states.clone()
    y, bottom = scans.run(form, rows, cols, gates, slots, states, lengths, heads, kv_heads, dim, vdim)
    y_walk, bottom_walk = scans.run(form, rows, cols, gates, slots, walked, lengths, heads, kv_heads, dim, vdim, chunk=0)
    pairs = [(y, y_walk), (states, walked)] + ([(bottom, bottom_walk)] if form == "memory" else [])
    scale = max(1.0, float(y_walk.abs().max()))
    assert all(float((a.double() - b.double()).abs().max()) <= 4e-5 * scale for a, b in pairs)


def distances(form, dtype, dim, vdim, length, kind, heads=4):
    """2-norm of the difference from float64 over that of the result: y (and the memory form's divisors), states.  Operands of either sign, positive
    ones, or small whole numbers whose decays are one."""
    rows, cols, gates, slots, states, kv_heads, columns = scans.problem(form, dtype, [length], heads, heads, dim, vdim, 31 + dim + length)
    if kind == "positive":
        rows, states = rows.abs(), states.abs()
    scale = 0.7
    if kind == "whole":
        rows, states, gates, scale = (rows.float() * 4).round().clamp(-2, 2).to(dtype), (states * 6).round(), torch.ones_like(gates), 1.0
    start = states[slots[0], 5:5 + heads * columns * dim].double().view(heads, columns, dim)
    y, bottom = scans.run(form, rows, cols, gates, slots, states, [length], heads, heads, dim, vdim, scale=scale)
    here = rows.double()
    q, k, v = (here[:, at:at + heads * size].view(length, heads, size) for at, size in zip(cols, (dim, dim, vdim)))
    keep = gates.double().expand(length, heads) if form == "decay" else gates.double()[:, :, 0]
    write = torch.ones_like(keep) if form == "decay" else gates.double()[:, :, 1]
    want, after = scans.recurrence(form, scale * q, k, v, keep, write, start)

    def off(found, exact):
        return float((found.double() - exact).norm() / exact.norm())

    found = [off(y, want[:, :, :vdim]), off(states[slots[0], 5:5 + heads * columns * dim], after.flatten())]
    if form == "memory":
        found[0] = max(found[0], off(bottom, torch.maximum(want[:, :, vdim].abs(), gates.double()[:, :, 2]) + 1e-6))
    return found


@pytest.mark.usefixtures("on_tensor_cores")
@pytest.mark.parametrize("kind,y_bound,state_bound", [("either sign", 0.9e-7, 0.65e-7), ("positive", 0.7e-7, 0.55e-7)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("form", ["memory", "decay"])
@pytest.mark.parametrize("dim,vdim", [(16, 64), (33, 40), (64, 128), (72, 96), (128, 256)])
@pytest.mark.parametrize("length", [33, 128, 300])
def test_distance_from_64_bits(form, dtype, dim, vdim, length, kind, y_bound, state_bound):
    """What is rounded once is off by 0.29 units of the last place (root mean square), 2.5e-8 of the number: a state is the sum of four such sums, which
    are smaller than it, and is rounded with each of them (a constant decay's powers are rounded alike in all of a head's numbers, which adds as
    much once more: 0.59e-7 with 64 columns); a row's scores are off by as much again, and its numbers by more where they have either sign.  What the
    sums in tensor memory drop, half a unit at each of several steps, would come on top of that (positive numbers without the decays' shares:
    y 0.86e-7 to 1.3e-7, states 0.59e-7 to 0.72e-7)."""
    y, state = distances(form, dtype, dim, vdim, length, kind)
    assert y <= y_bound and state <= state_bound


@pytest.mark.usefixtures("on_tensor_cores")
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("form", ["memory", "decay"])
@pytest.mark.parametrize("dim,vdim", [(6, 17), (64, 128), (128, 64)])
@pytest.mark.parametrize("length", [33, 300])
def test_small_whole_numbers_stay_exact(form, dtype, dim, vdim, length):
    """Decays and weights of one, sums below 2^24.  (The divisors have 1e-6 added to them: a rounding, 2^-24 of the number at most.)"""
    y, state = distances(form, dtype, dim, vdim, length, "whole")
    assert y <= (2.0 ** -24 if form == "memory" else 0.0) and state == 0.0


@pytest.mark.usefixtures("on_tensor_cores")
@pytest.mark.parametrize("form", ["memory", "delta", "decay"])
def test_an_infinity_reaches_no_token_before_it(form):
    scans.test_an_infinity_reaches_no_token_before_it(form)


@pytest.mark.usefixtures("on_tensor_cores")
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("form,which", [("memory", 0), ("memory", 1), ("memory", 2), ("decay", 2), ("delta", 0)])
@pytest.mark.parametrize("value", [float("inf"), float("nan"), 3.0e38])
def test_what_is_not_finite_is_summed_plainly(form, which, dtype, value):
    """One number of the queries, keys or values: the rows and matrices that it reaches are those of the walk, the others its to the bound."""
    lengths, bad = [300], 77
    rows, cols, gates, slots, states, kv_heads, columns = scans.problem(form, dtype, lengths, 2, 2, 72, 96, 21)
    rows[bad, cols[which] + 5] = value
    walked = states.clone()
    y, bottom = scans.run(form, rows, cols, gates, slots, states, lengths, 2, kv_heads, 72, 96)
    y_walk, bottom_walk = scans.run(form, rows, cols, gates, slots, walked, lengths, 2, kv_heads, 72, 96, chunk=0)
    usual = 30.0                                       # (results of the other numbers are below it; 3e38 times an ordinary number is not)
    # (An infinite query's own bottom is the floor in chunks, on either pipe: infinities of both signs meet in q n.)
    for a, b in [(y, y_walk), (states, walked)] + ([(bottom, bottom_walk)] if form == "memory" and which else []):
        small = b.abs() <= usual
        assert torch.equal(a.abs() <= usual, small)
        assert float((a - b).abs()[small].max()) <= 4e-5 * usual


def test_which_scans_run_there(monkeypatch):
    from miniserve_b200 import kernels

    taken = kernels._scanned_on_tensor_cores
    # memory and constant decay in bfloat16: always with more than 64 key entries, or enough work
    assert taken(256, 1, 256, 8, 128, 256, True) and not taken(512, 1, 512, 16, 64, 128, True) and taken(1000, 1, 1000, 16, 64, 128, True)
    # three parts: two tiles or two blocks, and more work
    assert not taken(256, 1, 256, 64, 128, 64, False) and taken(512, 1, 512, 64, 128, 64, False) and not taken(2048, 1, 2048, 32, 64, 64, False)
    # one value tile and one block; a memory form's tile of ones, and its own keys; the delta form's single block
    assert not taken(2048, 1, 2048, 16, 64, 64, True) and taken(2048, 1, 2048, 32, 64, 64, True)
    assert not taken(512, 1, 512, 64, 128, 64, False, "memory") and taken(2048, 1, 2048, 32, 128, 64, False, "memory")
    assert taken(512, 1, 512, 64, 96, 96, False, "memory") and not taken(1000, 1, 1000, 64, 64, 128, False, "memory")
    assert not taken(1000, 1, 1000, 32, 64, 128, False, "delta") and taken(2048, 1, 2048, 64, 64, 128, False, "delta")
    # portions that leave chunks empty
    assert not taken(2048, 30, 200, 8, 128, 256, True) and taken(2048, 20, 200, 8, 128, 256, True) and taken(1100, 65, 1036, 8, 128, 256, True)
    # records that do not fit: the float32 pipe's scratch
    n = 1_000_000
    assert len(kernels._chunk_scratch(n, 1, n, 8, 65, 9, "meta", tensor_cores=True)) == 2


def test_records_that_do_not_fit_leave_a_scan_to_the_float32_pipe(monkeypatch):
    """The scratch of either way is allowed, or of the float32 pipe's alone: which kernels run, and that those give what they give by themselves."""
    from miniserve_b200 import kernels

    monkeypatch.setattr(kernels, "CHUNK_SCAN_LONGEST", 0)
    rows, cols, gates, slots, states, kv_heads, columns = scans.problem("memory", torch.bfloat16, [300], 1, 1, 8, 8, 3)
    library, records, found = kernels.library(), [], []
    monkeypatch.setattr(library, "ms_chunk_scan", lambda *args, real=library.ms_chunk_scan: records.append(args[-3]) or real(*args))
    # floats of the pipe: five chunks' matrices and decays; of the tensor cores: three matrices, decays, three records
    limit = 4 * (5 * 9 * 8 + 5)
    for wanted, scratch in ((True, kernels.MAX_CHUNK_SCRATCH), (True, limit), (False, limit)):
        monkeypatch.setattr(kernels, "MAX_CHUNK_SCRATCH", scratch)
        monkeypatch.setattr(kernels, "_scanned_on_tensor_cores", lambda *args: wanted)
        kept = states.clone()
        y, bottom = scans.run("memory", rows, cols, gates, slots, kept, [300], 1, kv_heads, 8, 8)
        found.append((y, bottom, kept))
    assert records[0] and not records[1] and not records[2]
    assert all(torch.equal(a, b) for a, b in zip(found[1], found[2]))
    assert all(torch.allclose(a, b, rtol=4e-5, atol=4e-5) for a, b in zip(found[0], found[1]))
    kernels.check_device_errors(torch.device("cuda:0"))


@pytest.mark.usefixtures("on_tensor_cores")
@pytest.mark.parametrize("form,dtype", [("memory", torch.bfloat16), ("delta", torch.float32)])
def test_a_token_that_is_not_finite_costs_no_orders_of_magnitude(form, dtype):
    """A NaN in an early token's keys is in every later row and state: all of them are summed again, by whole blocks.  (Measured: 11 times the time without
    it; by a thread for each row and half a tile, 1,600 times.)"""
    lengths = [1000]
    rows, cols, gates, slots, states, kv_heads, columns = scans.problem(form, dtype, lengths, 8, 8, 128, 256, 17)
    times = []
    for value in (0.0, float("nan")):
        rows[3, cols[1]:cols[2]] = value
        for _ in range(3):
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            kept = states.clone()
            start.record()
            y, _ = scans.run(form, rows, cols, gates, slots, kept, lengths, 8, kv_heads, 128, 256)
            end.record()
            end.synchronize()
        times.append(start.elapsed_time(end))
    assert torch.isfinite(y[:3]).all() and not torch.isfinite(y[3:]).any()
    assert times[1] <= 30 * times[0]
