"""Which steps are scanned in chunks, with the rules in force, and steps that mix portions with decoded tokens: those are walked beside the
scan, as they are in a step of their own."""

import importlib

import helpers
import pytest
import torch

from test_chunk_scan_gpu import ints, problem, recurrence, run

pytestmark = pytest.mark.gpu

MIXED = [[310] + [1] * 40, [1, 31, 32, 33, 400, 0, 2], [1] * 33 + [260, 5, 700, 1]]


def counted(monkeypatch, *names):
    from miniserve_b200 import kernels

    lib, calls = kernels.library(), dict.fromkeys(names, 0)
    for name in names:
        def wrapped(*args, _name=name, _real=getattr(lib, name)):
            calls[_name] += 1
            return _real(*args)
        monkeypatch.setattr(lib, name, wrapped)
    return calls


@pytest.mark.parametrize("form", ["memory", "delta", "decay"])
@pytest.mark.parametrize("lengths", MIXED)
def test_matrix_scan(monkeypatch, form, lengths):
    if form == "delta":
        lengths = [3 * length if length >= 256 else length for length in lengths]      # (its rule asks for longer portions)
    heads, kv_heads, dim, vdim = 4, 2, 64, 80
    rows, cols, gates, slots, states, kv_heads, columns = problem(form, torch.bfloat16, lengths, heads, kv_heads, dim, vdim, 7)
    walked = states.clone()
    calls = counted(monkeypatch, "ms_chunk_scan", "ms_matrix_scan")
    y, bottom = run(form, rows, cols, gates, slots, states, lengths, heads, kv_heads, dim, vdim)
    assert calls == {"ms_chunk_scan": 1, "ms_matrix_scan": 1}
    y_walk, bottom_walk = run(form, rows, cols, gates, slots, walked, lengths, heads, kv_heads, dim, vdim, chunk=0)
    assert calls == {"ms_chunk_scan": 1, "ms_matrix_scan": 2}
    scale, at = max(1.0, float(y_walk.abs().max())), 0
    for r, length in enumerate(lengths):
        pairs = [(y[at:at + length], y_walk[at:at + length]), (states[slots[r]], walked[slots[r]])]
        if form == "memory":
            pairs.append((bottom[at:at + length], bottom_walk[at:at + length]))
        for a, b in pairs:                                  # (either way is within 2e-5 of the definition)
            assert torch.equal(a, b) if length < 32 else float((a - b).abs().max()) <= 4e-5 * scale
        assert length < 32 or not torch.equal(states[slots[r]], walked[slots[r]])
        at += length


@pytest.mark.parametrize("lengths", MIXED)
def test_selective_scan(monkeypatch, lengths):
    from miniserve_b200 import kernels

    heads, P, N, G = 4, 64, 96, 2
    g = torch.Generator(device="cuda").manual_seed(len(lengths))
    n, inner = sum(lengths), heads * P
    conv = torch.randn((n, inner + 2 * G * N), generator=g, device="cuda") * 0.5
    proj = (torch.randn((n, heads), generator=g, device="cuda") * 2).bfloat16()
    dt_bias, a_log, skip = (torch.randn(heads, generator=g, device="cuda") for _ in range(3))
    slots = torch.randperm(len(lengths), generator=g, device="cuda")
    start = torch.randn((len(lengths), inner * N), generator=g, device="cuda") * 0.3
    calls = counted(monkeypatch, "ms_selective_chunk_scan", "ms_selective_scan")

    def scan(tokens, requests, **options):
        """The rows of y and the states of a step of these requests (their tokens given)."""
        states, y = start.clone(), torch.full((len(tokens), inner), float("nan"), device="cuda")
        own = [lengths[r] for r in requests]
        kernels.selective_scan(conv[tokens], proj[tokens], 0, dt_bias, a_log, skip, states, 0, slots[requests].to(torch.int32),
                               ints([sum(own[:i]) for i in range(len(own) + 1)]), heads, P, N, G, y, max_query_len=max(own), **options)
        return y, states

    request_of = [r for r, length in enumerate(lengths) for _ in range(length)]
    everything, short = list(range(len(lengths))), [r for r, length in enumerate(lengths) if length < 32]
    short_tokens = [t for t in range(n) if lengths[request_of[t]] < 32]
    long_tokens = [t for t in range(n) if lengths[request_of[t]] >= 32]
    y, states = scan(list(range(n)), everything)
    assert calls == {"ms_selective_chunk_scan": 1, "ms_selective_scan": 1}
    y_alone, alone = scan(short_tokens, short)
    assert torch.equal(y[short_tokens], y_alone) and torch.equal(states[slots[short]], alone[slots[short]])
    y_walk, walked = scan(list(range(n)), everything, chunked=False)
    assert calls == {"ms_selective_chunk_scan": 1, "ms_selective_scan": 3}
    scale = max(1.0, float(y_walk.abs().max()))             # (either way is within 2e-5 of the definition)
    assert float((y - y_walk)[long_tokens].abs().max()) <= 4e-5 * scale and float((states - walked).abs().max()) <= 4e-5 * scale


@pytest.mark.parametrize("lengths,delta,taken,walk_beside", [
    ([255], False, False, False), ([256], False, True, False), ([127, 385], False, True, False), ([127] * 5, False, False, False),
    ([128] * 4, False, True, False), ([300, 200, 100], False, True, True), ([128] * 3 + [127], False, False, False), ([256, 32], False, True, False), ([256, 31], False, True, True),
    ([256] + [1] * 28, False, True, True), ([256] + [1] * 29, False, False, False), ([327] + [1] * 64, False, False, False), ([328] + [1] * 64, False, True, True),
    ([255], True, False, False), ([256], True, True, False), ([383, 1], True, False, False), ([384, 1], True, True, True),
    ([500] * 4, True, False, False), ([640] * 4, True, True, False)])
def test_which_steps_are_scanned_in_chunks(monkeypatch, lengths, delta, taken, walk_beside):
    """256 tokens, or 128 in a step of 512; the delta form 128 (1 + portions of that length that the step would fill).  Of more than two
    unequal portions one may be too short for a chunk, as far as the host knows: the walk is launched beside the scan then.  More
    than 28 requests that are too short ask for a longer portion, two tokens each."""
    form = "delta" if delta else "memory"
    rows, cols, gates, slots, states, kv_heads, columns = problem(form, torch.bfloat16, lengths, 1, 1, 8, 8, 3)
    calls = counted(monkeypatch, "ms_chunk_scan", "ms_matrix_scan")
    run(form, rows, cols, gates, slots, states, lengths, 1, kv_heads, 8, 8)
    assert calls == {"ms_chunk_scan": int(taken), "ms_matrix_scan": int(walk_beside or not taken)}


@pytest.mark.parametrize("N", [32, 64, 96, 128, 160, 192, 224, 256])
@pytest.mark.parametrize("lengths", [[1] * 5, [7, 1], [40]])
def test_the_walk_with_states_of_any_multiple_of_32(N, lengths):
    """A lane has 1, 2, 4 or 8 entries of a column: states of 96, 160, 192 and 224 numbers leave some of them empty."""
    from miniserve_b200 import kernels

    heads, P, G = 2, 32, 1
    g = torch.Generator(device="cuda").manual_seed(N)
    n, inner = sum(lengths), heads * P
    conv = torch.randn((n, inner + 2 * G * N), generator=g, device="cuda") * 0.5
    proj = torch.randn((n, heads), generator=g, device="cuda").bfloat16()
    dt_bias, a_log, skip = (torch.randn(heads, generator=g, device="cuda") for _ in range(3))
    start = torch.randn((len(lengths), inner * N), generator=g, device="cuda") * 0.3
    states, y = start.clone(), torch.full((n, inner), float("nan"), device="cuda")
    starts = [sum(lengths[:r]) for r in range(len(lengths) + 1)]
    kernels.selective_scan(conv, proj, 0, dt_bias, a_log, skip, states, 0, ints(list(range(len(lengths)))), ints(starts), heads, P, N, G, y,
                           max_query_len=max(lengths), chunked=False)
    for r, length in enumerate(lengths):
        here, rows = conv[starts[r]:starts[r + 1]].double(), slice(starts[r], starts[r + 1])
        b, c = (here[:, at:at + N].view(length, 1, N).repeat_interleave(heads, 1) for at in (inner, inner + N))
        x = here[:, :inner].view(length, heads, P)
        dt = torch.nn.functional.softplus(proj[rows].double() + dt_bias.double())
        want, after = recurrence("ssm", c, b, x, torch.exp(-torch.exp(a_log.double()) * dt), dt, start[r].double().view(heads, P, N))
        want = (want + skip.double()[:, None] * x).reshape(length, inner)
        scale = max(1.0, float(want.abs().max()))
        assert float((y[rows].double() - want).abs().max()) <= 2e-5 * scale                 # (the walk's bound, as above)
        assert float((states[r].double() - after.flatten()).abs().max()) <= 2e-5 * scale


@pytest.mark.parametrize("form,heads,dim,columns,most", [("memory", 8, 128, 257, 65215), ("delta", 16, 128, 128, 26196), ("decay", 16, 128, 128, 65471)])
def test_beyond_a_gibibyte_of_scratch_a_scan_walks(form, heads, dim, columns, most):
    """All of a form's scratch counts: the delta form's W, U and keys are more than its chunks' matrices."""
    from miniserve_b200 import kernels

    for n in (most, most + 200):
        scratch = kernels._chunk_scratch(n, 1, n, heads, dim, columns, "meta", form == "delta")
        assert (scratch is None) is (n > most)
        assert scratch is None or sum(4 * t.numel() for t in scratch) <= 1 << 30


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("design,name,scan,walk", [("kivurax", "c", "ms_chunk_scan", "ms_matrix_scan"), ("kivurax", "d", "ms_chunk_scan", "ms_matrix_scan"),
                                                   ("zozezen", "c", "ms_selective_chunk_scan", "ms_selective_scan")])
def test_a_long_prompt_beside_decoded_tokens_of_a_model(tmp_path, monkeypatch, dtype, design, name, scan, walk):
    """A step of the whole engine: 430 tokens of one prompt and the next token of each of nine requests, every logit against the plain
    whole-sequence computation, before and after it too."""
    tests, parts = importlib.import_module(f"test_{design}_gpu"), importlib.import_module(f"{design}_helpers")
    folder = parts.make_folder(tmp_path, name, seed=21)
    vocab = parts.CONFIGS[name]["vocab"]
    short = {f"s{i}": helpers.random_tokens(vocab, n, seed=30 + i) for i, n in enumerate((3, 5, 9, 17, 18, 33, 40, 65, 7))}
    requests = dict(short, long=helpers.random_tokens(vocab, 432, seed=50))
    steps = [dict(step=0, entries=[dict(id=rid, tokens=t[:-2], want=list(range(len(t) - 2))) for rid, t in short.items()], end=[]),
             dict(step=1, entries=[dict(id="s0", tokens=short["s0"][-2:-1], want=[0]), dict(id="long", tokens=requests["long"][:430], want=list(range(430)))]
                  + [dict(id=rid, tokens=t[-2:-1], want=[0]) for rid, t in list(short.items())[1:]], end=[]),
             dict(step=2, entries=[dict(id="long", tokens=requests["long"][430:], want=[0, 1])]
                  + [dict(id=rid, tokens=t[-1:], want=[0]) for rid, t in short.items()], end=list(requests))]
    runtime = tests.build(folder, dtype, 120, 8, max_seqs=10)
    calls = counted(monkeypatch, scan, walk)
    got = helpers.collect(steps, tests.replay(runtime, steps))
    tests.check(folder, dtype, requests, got)
    assert calls[scan] >= 1 and calls[walk] >= 3 * calls[scan]         # (a layer walks in all three steps, beside the scan in the second)
