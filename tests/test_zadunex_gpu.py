"""Zadunex on the GPU: every mechanism's kernels alone against the plain functions of
tests/plain_zadunex.py, then the model through the engine: whole prompts, portions, single tokens,
unequal batches, reused slots, far tokens, long decoding, greedy generation and trace replay."""

import io
import json
import math
from types import SimpleNamespace

import pytest
import torch

import plain_zadunex as plain
from zadunex_helpers import CONFIGS, assert_logits, plain_logits, prompts, write_folder

pytestmark = pytest.mark.gpu

DTYPES = (torch.float32, torch.bfloat16)
PART_TOL = {torch.float32: 3e-5, torch.bfloat16: 5e-2}


@pytest.fixture(scope="module")
def folders(tmp_path_factory):
    root = tmp_path_factory.mktemp("zadunex_gpu")
    return {name: write_folder(root / name, name) for name in CONFIGS}


def runtime(dtype):
    from kernel_rush_kawk_b200.csrc import load_kernels
    from kernel_rush_kawk_b200.engine.model import Runtime

    return Runtime(torch.device("cuda:0"), dtype, load_kernels((16, 32)))


def rand(shape, seed, scale=1.0):
    g = torch.Generator().manual_seed(seed)
    return torch.randn(shape, generator=g) * scale


def context(rt, slots, starts, q_lens, cache):
    from kernel_rush_kawk_b200.engine.step import BatchMeta, StepContext

    meta = BatchMeta(sum(q_lens), len(slots), 0, rt.device)
    meta.fill(slots, starts, [[0] * n for n in q_lens], [])
    return StepContext(rt.ops, meta, cache)


def close(got, ref, dtype, what):
    got, ref = got.detach().double().cpu(), ref.detach().double().cpu()
    assert got.shape == ref.shape, f"{what}: shape {tuple(got.shape)} vs {tuple(ref.shape)}"
    assert torch.isfinite(got).all(), f"{what}: non-finite values"
    err = (got - ref).abs().max().item()
    tol = PART_TOL[dtype] * ref.abs().max().item()
    assert err <= tol, f"{what}: max |d| = {err:.3e} > {tol:.3e}; first bad row {int(((got - ref).abs() > tol).any(-1).nonzero()[0])}"


def run_part(part, rt, h, pieces, dtype, prior=()):
    """One sequence through a mixer part, cut into ``pieces``; ``prior``: sequences that used (and gave
    back) the slot before."""
    from kernel_rush_kawk_b200.cache import SequenceCache

    cache = SequenceCache([part.cache_need()], 2048, 1, 2048, rt.device, dtype)
    for seq, cuts in list(prior) + [(h, pieces)]:
        slot = cache.alloc()
        got, start = [], 0
        for n in cuts:
            cache.reserve(slot, start + n)
            cache.sync()
            ctx = context(rt, [slot], [start], [n], cache)
            got.append(part.forward(ctx, seq[start:start + n].to(dtype).cuda(), cache.view(0)))
            cache.advance(slot, n)
            start += n
        cache.free(slot)
    rt.ops.check()
    return torch.cat(got)


def as_path(w, dtype):
    """The tensors as the path stores them, and the same values in float64 for the plain functions."""
    stored = {k: v.to(torch.bfloat16) for k, v in w.items()}  # checkpoints hold bfloat16
    return {k: v.to(dtype).cuda() for k, v in stored.items()}, {k: v.double() for k, v in stored.items()}


# ----------------------------------------------------------------------------------------------
# each mechanism alone
# ----------------------------------------------------------------------------------------------

@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("streams, width", [(1, 72), (2, 64), (3, 50), (4, 33), (8, 16)])
def test_hyper_connection_norm_folds_reads_and_normalises(dtype, streams, width):
    """Two sublayers in a row: the first norm only reads; the second writes the first sublayer's output back
    through its M and b, reads through its own a, and leaves its own M and b on the stream."""
    from kernel_rush_kawk_b200.parts import HyperRMSNorm, Stream

    rt = runtime(dtype)
    ctx = SimpleNamespace(ops=rt.ops)
    S, C, rows = streams, width, 7
    X = rand((rows, S, C), 1, 3.0)
    norms, ws = [], []
    for q in range(2):
        w = {"weight": (1 + 0.3 * rand((C,), 10 + q)), "in": rand((S,), 20 + q), "out": rand((S,), 30 + q),
             "mix": rand((S, S), 40 + q)}
        part = HyperRMSNorm({"size": C, "eps": 1e-4, "streams": S})
        assert {k: tuple(s.shape) for k, s in part.tensor_specs().items()} == {k: tuple(v.shape) for k, v in w.items()}
        dev, ref = as_path(w, dtype)
        part.bind(dev, rt)
        norms.append(part)
        ws.append(ref)
    stream = Stream(X.reshape(rows, S * C).cuda())
    h1 = norms[0].forward(ctx, stream).tensor()
    Xd = X.double()
    close(h1, plain.rms_norm(torch.einsum("s,rsc->rc", ws[0]["in"], Xd), ws[0]["weight"], 1e-4), dtype, "first read")
    assert stream.branch is None and stream.fold is not None
    y = rand((rows, C), 5, 2.0).to(dtype)
    stream.branch = y.cuda()
    h2 = norms[1].forward(ctx, stream).tensor()
    X2 = torch.einsum("st,rsc->rtc", ws[0]["mix"], Xd) + ws[0]["out"][None, :, None] * y.double()[:, None, :]
    assert (stream.x.double().cpu().view(rows, S, C) - X2).abs().max() < 1e-4  # the streams are 32-bit whatever the path
    close(h2, plain.rms_norm(torch.einsum("s,rsc->rc", ws[1]["in"], X2), ws[1]["weight"], 1e-4), dtype, "fold and read")
    last = HyperRMSNorm({"size": C, "eps": 1e-4, "streams": S, "read": "sum"})
    last.bind({"weight": ws[0]["weight"].to(dtype).cuda()}, rt)
    stream.branch = y.cuda()
    h3 = last.forward(ctx, stream).tensor()
    X3 = torch.einsum("st,rsc->rtc", ws[1]["mix"], X2) + ws[1]["out"][None, :, None] * y.double()[:, None, :]
    close(h3, plain.rms_norm(X3.sum(dim=1), ws[0]["weight"], 1e-4), dtype, "the sum of the streams")


SSM_SHAPES = [  # hidden, heads, head_dim, state, groups, taps, norm parts
    (64, 4, 16, 24, 2, 4, 2),
    (48, 2, 32, 16, 1, 3, 1),
    (50, 3, 10, 7, 3, 4, 2),
    (32, 1, 64, 8, 1, 5, 4),
    (40, 6, 8, 40, 6, 2, 3),
    (32, 2, 12, 5, 2, 1, 1),
    (64, 2, 64, 128, 1, 4, 1),   # a head of 64 x 128: thirty-two rows of the state a lane
    (32, 2, 4, 200, 2, 4, 8),    # narrow heads and a long state: every lane of a warp on one column
]


def ssm_part(shape, dtype, rt, seed=50):
    from kernel_rush_kawk_b200.parts import Mamba2

    C, H, P, N, G, taps, parts = shape
    inner, ch = H * P, H * P + 2 * G * N
    m = {"heads": H, "vdim": P, "state": N, "groups": G, "conv": taps, "norm_groups": parts}
    part = Mamba2({"hidden": C, "heads": H, "head_dim": P, "state": N, "groups": G, "taps": taps, "norm_groups": parts,
                   "eps": 1e-5})
    w = {"in": rand((2 * inner + 2 * G * N + H, C), seed + 1, 0.25), "conv": rand((ch, taps), seed + 2, 0.4),
         "conv.b": rand((ch,), seed + 3, 0.2), "dt_bias": rand((H,), seed + 4, 1.0) - 0.5,
         "A_log": rand((H,), seed + 5, 1.0) - 2.5, "D": 1 + rand((H,), seed + 6, 0.3),
         "norm": 1 + rand((inner,), seed + 7, 0.2), "o": rand((C, inner), seed + 8, 0.2)}
    assert {k: tuple(s.shape) for k, s in part.tensor_specs().items()} == {k: tuple(v.shape) for k, v in w.items()}
    dev, ref = as_path(w, dtype)
    part.bind(dev, rt)
    return part, m, ref


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("shape", SSM_SHAPES)
def test_state_space_mixer_alone(dtype, shape):
    """Whole (long enough for the scan in chunks), in pieces down to two tokens and fewer than the
    convolution's taps, token by token, and in a slot whose state another sequence left."""
    rt = runtime(dtype)
    part, m, ref = ssm_part(shape, dtype, rt)
    T = 300
    h = rand((T, shape[0]), 11).to(dtype)
    want = plain.mamba2(h.double(), ref, "", m, 1e-5)
    other = rand((70, shape[0]), 12).to(dtype)
    for pieces, prior in (([T], ()), ([127, 2, 1, 3, 129, 38], ()), ([270] + [1] * 30, ()), ([T], [(other, [69, 1])])):
        got = run_part(part, rt, h, pieces, dtype, prior=prior)
        close(got, want, dtype, f"state-space mixer {shape}, pieces {pieces[:4]}, prior {len(prior)}")


def ssd_in_64_bits(x, B, C, dt, bias, a_log, skip, groups, lens, start):
    rows, H = dt.shape
    d = torch.nn.functional.softplus(dt.double() + bias.double())
    decay = torch.exp(-torch.exp(a_log.double()) * d)
    xx, per = x.double().view(rows, H, -1), H // groups
    bb, cc = (t.double().view(rows, groups, -1).repeat_interleave(per, 1) for t in (B, C))
    y, states, row = torch.empty_like(xx), [], 0
    for i, n in enumerate(lens):
        S = start[i].double()
        for t in range(row, row + n):
            S = decay[t][:, None, None] * S + (d[t][:, None] * bb[t])[:, :, None] * xx[t][:, None, :]
            y[t] = torch.einsum("hn,hnp->hp", cc[t], S) + skip.double()[:, None] * xx[t]
        states.append(S)
        row += n
    return y.view(rows, -1), torch.stack(states)


@pytest.mark.parametrize("rate", [-6.0, 0.0, 3.0, "trained"])
@pytest.mark.parametrize("lens", [[96], [131, 64, 1, 33], [300, 65]])
@pytest.mark.parametrize("shape", [(4, 64, 128, 2), (3, 80, 16, 1), (2, 16, 48, 2)])  # heads, head size, state rows, groups
def test_state_space_scans_on_the_tensor_cores(shape, lens, rate, monkeypatch):
    """Chunks of 64 tokens, whole and in portions of one chunk (little scratch), from a state that is not zero, with decays
    from almost none to everything within a token: outputs and state no further from 64 bits than twice what the scan
    token by token is (and 2e-7, a few roundings at 2^-24)."""
    rt = runtime(torch.bfloat16)
    H, P, N, G = shape
    rows = sum(lens)
    buf = rand((rows, H * P + 2 * G * N), 31).to(torch.bfloat16).cuda()
    x, B, C = buf[:, :H * P], buf[:, H * P:H * P + G * N], buf[:, H * P + G * N:]
    dt, bias = rand((rows, H), 32).to(torch.bfloat16).cuda(), rand((H,), 33).cuda()
    a_log, skip = rand((H,), 34, 0.3).cuda(), rand((H,), 35).cuda()
    if rate == "trained":  # rates of 1 to 16, steps of 0.001 to 0.1
        a_log, dt = torch.linspace(0.0, 2.77, H).cuda(), dt * 0.2
        bias = torch.log(torch.expm1(torch.exp(torch.linspace(-2.3, -6.9, H)))).cuda()
    else:
        a_log += rate
    start = rand((len(lens), H, N, P), 36).cuda()
    want, want_state = ssd_in_64_bits(x, B, C, dt, bias, a_log, skip, G, lens, start)
    ctx = context(rt, list(range(len(lens))), [0] * len(lens), lens, None)
    off = {}
    for name, least, scratch in (("tokens", 1 << 30, 1 << 28), ("chunks", 1, 1 << 28), ("portions", 1, 1)):
        monkeypatch.setattr(type(rt.ops), "SSD_TENSOR_MIN", least)
        monkeypatch.setattr(type(rt.ops), "SSD_SCRATCH", scratch)
        state = start.clone()
        y = rt.ops.ssd_scan(x, B, C, dt, bias, a_log, skip, H, P, N, G, state, ctx.batch)
        off[name] = [((a.double() - b).norm() / b.norm()).item() for a, b in ((y, want), (state, want_state))]
        if name == "chunks":
            whole = y, state
    assert torch.equal(y, whole[0]) and torch.equal(state, whole[1]), "portions are the same sums"
    assert all(c <= 2 * t + 2e-7 for c, t in zip(off["chunks"], off["tokens"])), off


@pytest.mark.parametrize("shape, lens", [
    ((48, 64, 128, 4), [450]),            # more blocks than the SMs hold two of, not more than three
    ((48, 64, 128, 4), [600, 400, 300]),  # several heads a block, sequences that end before others
    ((24, 80, 32, 2), [1100]),            # a head's second slice of columns in the block of the first
    ((40, 64, 272, 2), [700]),            # more rows of the state than are fetched at a time
])
def test_state_space_scans_of_many_heads(shape, lens, monkeypatch):
    """Enough heads and chunks that a block takes several units of a group's chunk one after the other, or that three share an SM: from 64
    bits no further than twice the scan token by token, portions the same bits, and an infinite value of one head reaches no earlier
    token, no other column and no other head."""
    rt = runtime(torch.bfloat16)
    H, P, N, G = shape
    rows = sum(lens)
    x, B, C = (rand((rows, n), 61 + i).to(torch.bfloat16).cuda() for i, n in enumerate((H * P, G * N, G * N)))
    dt, bias = rand((rows, H), 64).to(torch.bfloat16).cuda(), rand((H,), 65).cuda() - 2
    a_log, skip = rand((H,), 66, 0.5).cuda(), rand((H,), 67).cuda()
    start = rand((len(lens), H, N, P), 68).cuda()
    ctx = context(rt, list(range(len(lens))), [0] * len(lens), lens, None)

    def scan(x, least, scratch=1 << 28):
        monkeypatch.setattr(type(rt.ops), "SSD_TENSOR_MIN", least)
        monkeypatch.setattr(type(rt.ops), "SSD_SCRATCH", scratch)
        state = start.clone()
        return rt.ops.ssd_scan(x, B, C, dt, bias, a_log, skip, H, P, N, G, state, ctx.batch), state

    want = ssd_in_64_bits(x, B, C, dt, bias, a_log, skip, G, lens, start)
    tokens, chunks, portions = scan(x, 1 << 30), scan(x, 1), scan(x, 1, 12 * start.numel())  # three chunks at a time
    assert all(torch.equal(a, b) for a, b in zip(chunks, portions))
    off = lambda got: [((a.double() - b).norm() / b.norm()).item() for a, b in zip(got, want)]
    assert all(c <= 2 * t + 2e-7 for c, t in zip(off(chunks), off(tokens))), (off(chunks), off(tokens))
    at, col = 250, 3 * P + 5  # the fourth head
    x[at, col] = float("-inf")
    y, state = scan(x, 1)
    rest = [c for c in range(H * P) if c != col]
    assert torch.equal(y[:at], chunks[0][:at]) and torch.equal(y[:, rest], chunks[0][:, rest]) and not torch.isfinite(y[at:lens[0], col]).any()
    clean = torch.ones_like(start, dtype=torch.bool)
    clean[0, 3, :, 5] = False
    assert torch.equal(state[clean], chunks[1][clean]) and not torch.isfinite(state[~clean]).any()


def test_step_sizes_of_a_prompt_of_millions(monkeypatch):
    """4,194,305 tokens of one head are 65,537 chunks, more than a grid has rows: their step sizes and summed decays all the same (the scan itself
    goes through them in portions)."""
    rt = runtime(torch.bfloat16)
    rows, L = 65536 * 64 + 1, 64
    dt = torch.linspace(-3, 1, 64).repeat(65537)[:rows].to(torch.bfloat16).cuda()
    one = torch.zeros(1, device="cuda")
    steps = torch.empty((rows, 4), dtype=torch.float32, device="cuda")
    cu, qlen = (torch.tensor(t, dtype=torch.int32, device="cuda") for t in ([0, rows], [rows]))
    rt.ops._ok(rt.ops.memory.krk_ssd_steps(steps.data_ptr(), dt.data_ptr(), 1, one.data_ptr(), one.data_ptr(), rows, 1, 1, rows, cu.data_ptr(),
                                           qlen.data_ptr(), rt.ops._stream()), "step sizes and decays")
    whole = steps[:-1].view(-1, L, 4)
    d = torch.nn.functional.softplus(dt[:L].float())
    assert torch.equal(whole, whole[:1].expand_as(whole))
    assert ((steps[:L, 2] - d).abs() <= 1e-6 * d).all() and ((steps[-1, 2] - d[0]).abs() <= 1e-6 * d[0]) and torch.isfinite(steps[-1]).all()
    assert torch.equal(steps[-1, 2:3], steps[-1, 3:]), "the last token's weight is its step size: nothing comes after it"


def test_a_state_space_token_after_its_decay(monkeypatch):
    """One token in front of a chunk, alone: what is left of it later in the chunk is e^d times it, d the difference of two sums of 64
    bits rounded once, so off by a rounding of d: a unit of its last place over the root of 12. A difference rounded twice would be off by
    the root of 2 more. Beside it e^ and the products are rounded to 2^-24 each: of d between 16 and 32 a twentieth."""
    rt = runtime(torch.bfloat16)
    monkeypatch.setattr(type(rt.ops), "SSD_TENSOR_MIN", 1)
    H, P, N, rows = 64, 16, 16, 64
    x, B, C = torch.zeros((rows, H * P)), torch.zeros((rows, N)), torch.zeros((rows, N))
    x[3], B[3, 0], C[:, 0] = 1.0, 1.0, 1.0
    x, B, C = (t.to(torch.bfloat16).cuda() for t in (x, B, C))
    dt = rand((rows, H), 71, 0.3).to(torch.bfloat16).cuda()
    bias, a_log, skip = rand((H,), 72).cuda(), torch.zeros(H, device="cuda"), torch.zeros(H, device="cuda")
    state = torch.zeros((1, H, N, P), device="cuda")
    ctx = context(rt, [0], [0], [rows], None)
    y = rt.ops.ssd_scan(x, B, C, dt, bias, a_log, skip, H, P, N, 1, state, ctx.batch).view(rows, H, P)[:, :, 0].double()
    d = torch.nn.functional.softplus(dt.float() + bias)  # the step sizes and log decays are numbers of 32 bits
    f = -(torch.exp(a_log) * d).double().cumsum(0)
    want = torch.exp(f - f[3]) * d[3].double()
    seen = (f - f[3] < -16) & (f - f[3] > -32)
    assert seen.sum() > 900
    off = ((y - want) / want)[seen].pow(2).mean().sqrt().item()
    # the kernel's own softplus may differ from torch's by a unit or two of 2^-24, which moves d by as much again
    assert off < 1.2 * 2.0 ** -19 / 12 ** 0.5, off


@pytest.mark.parametrize("dtype", DTYPES)
def test_convolution_of_many_rows(dtype, monkeypatch):
    """Rows in runs of eight a thread, four taps: sequences that start anywhere in a run, shorter than the taps, channels
    that fill no block. The same bits as the kernel of single elements, which rows off a 16-byte boundary take."""
    rt = runtime(dtype)
    monkeypatch.setattr(type(rt.ops), "_conv_walks", lambda *_: True)
    ch, lens = 520, [15, 1, 2, 33, 48, 7]
    rows = sum(lens)
    x = rand((rows, ch), 50).to(dtype).cuda()
    odd = torch.empty((rows, ch + 1), dtype=dtype, device="cuda")
    odd[:, 1:] = x
    w, b, tail = rand((4, ch), 51).cuda(), rand((ch,), 52).cuda(), rand((7, 3, ch), 53).to(dtype).cuda()
    ctx = context(rt, [1, 0, 4, 3, 5, 6], [9] * 6, lens, None)
    tails = [tail.clone(), tail.clone()]
    got = rt.ops.causal_conv_silu(x, w, b, tails[0], ctx.batch)
    want = rt.ops.causal_conv_silu(odd[:, 1:], w, b, tails[1], ctx.batch)
    assert torch.equal(got, want) and torch.equal(tails[0], tails[1])


@pytest.mark.parametrize("walks", [True, False])
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("lens", [[1] * 70, [1] * 64 + [500], [15, 1, 2, 33, 48, 7], [3, 17, 300, 1, 16, 64]])
def test_convolution_rows_in_runs_and_one_by_one(dtype, lens, walks, monkeypatch):
    """Whichever kernel a step takes: the same bits as the kernel of single elements, outputs and stored inputs, with sequences that start
    anywhere in a thread's eight rows."""
    rt = runtime(dtype)
    monkeypatch.setattr(type(rt.ops), "_conv_walks", lambda *_: walks)
    ch, rows = 520, sum(lens)
    x = rand((rows, ch), 50).to(dtype).cuda()
    odd = torch.empty((rows, ch + 1), dtype=dtype, device="cuda")
    odd[:, 1:] = x
    w, b, tail = rand((4, ch), 51).cuda(), rand((ch,), 52).cuda(), rand((len(lens), 3, ch), 53).to(dtype).cuda()
    ctx = context(rt, list(range(len(lens)))[::-1], [9] * len(lens), lens, None)
    tails = [tail.clone(), tail.clone()]
    got = rt.ops.causal_conv_silu(x, w, b, tails[0], ctx.batch)
    want = rt.ops.causal_conv_silu(odd[:, 1:], w, b, tails[1], ctx.batch)
    assert torch.equal(got, want) and torch.equal(tails[0], tails[1])


def test_convolution_of_more_runs_of_rows_than_a_grid_has(monkeypatch):
    """A step of 524,300 rows, 65,538 runs of eight: the same bits as a block a row."""
    rt = runtime(torch.bfloat16)
    ch, lens = 8, [524000, 300]
    x = rand((sum(lens), ch), 50).to(torch.bfloat16).cuda()
    w, b, tail = rand((4, ch), 51).cuda(), rand((ch,), 52).cuda(), rand((2, 3, ch), 53).to(torch.bfloat16).cuda()
    batch = SimpleNamespace(n_seqs=2, row_seq=torch.repeat_interleave(torch.arange(2), torch.tensor(lens)).int().cuda(),
                            cu_q=torch.tensor([0, lens[0], sum(lens)], dtype=torch.int32, device="cuda"),
                            seq_qlen=torch.tensor(lens, dtype=torch.int32, device="cuda"), seq_slot=torch.tensor([1, 0], dtype=torch.int32, device="cuda"))
    runs = []
    for walks in (True, False):
        monkeypatch.setattr(type(rt.ops), "_conv_walks", lambda *_, walks=walks: walks)
        stored = tail.clone()
        runs.append((rt.ops.causal_conv_silu(x, w, b, stored, batch), stored))
    assert all(torch.equal(a, b) for a, b in zip(*runs))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("n", [4, 32, 124, 256, 260, 768, 772, 1024, 1028])
def test_gated_norm_of_parts_of_any_size(dtype, n):
    """Up to 1,024 elements a part a warp each, beyond that a block: within an element's rounding and a sum's of n terms."""
    rt = runtime(dtype)
    rows, parts = 5, 3
    y, z = rand((rows, parts * n), 54).cuda(), rand((rows, parts * n), 55).to(dtype).cuda()
    weight, out = (1 + rand((parts * n,), 56, 0.2)).cuda(), torch.zeros((rows, parts * n + 8), dtype=dtype, device="cuda")
    rt.ops.gated_group_norm(y, z, weight, parts, 1e-5, out, 4, 0.5)
    v = (y.double() * torch.nn.functional.silu(z.double())).view(rows, parts, n)
    want = 0.5 * (v / torch.sqrt((v * v).mean(-1, keepdim=True) + 1e-5)).view(rows, -1) * weight.double()
    unit = 2.0 ** -8 if dtype == torch.bfloat16 else 2e-6
    assert ((out[:, 4:-4].double() - want).abs() <= unit * want.abs() + 1e-12).all()
    assert not out[:, :4].any() and not out[:, -4:].any()


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("n", [4, 124, 256, 260, 768, 772, 1024])
def test_gated_norm_of_many_parts(dtype, n):
    """Enough parts for a warp each, and one row less than fills the last block of eight: within an element's rounding and a
    sum's of n terms."""
    rt = runtime(dtype)
    rows, parts = 685, 3
    assert rt.ops._norm_by_warps(rows * parts, n)
    y, z = rand((rows, parts * n), 54).cuda(), rand((rows, parts * n), 55).to(dtype).cuda()
    weight, out = (1 + rand((parts * n,), 56, 0.2)).cuda(), torch.zeros((rows, parts * n + 8), dtype=dtype, device="cuda")
    rt.ops.gated_group_norm(y, z, weight, parts, 1e-5, out, 4, 0.5)
    v = (y.double() * torch.nn.functional.silu(z.double())).view(rows, parts, n)
    want = 0.5 * (v / torch.sqrt((v * v).mean(-1, keepdim=True) + 1e-5)).view(rows, -1) * weight.double()
    unit = 2.0 ** -8 if dtype == torch.bfloat16 else 2e-6
    assert ((out[:, 4:-4].double() - want).abs() <= unit * want.abs() + 1e-12).all()
    assert not out[:, :4].any() and not out[:, -4:].any()


@pytest.mark.parametrize("walks", [True, False])
@pytest.mark.parametrize("dtype", DTYPES)
def test_silu_of_the_most_negative(dtype, walks, monkeypatch):
    """Down to where e^-z still is a number: 1e-36 is as exact as any other result of the convolution and of the gated norm."""
    rt = runtime(dtype)
    monkeypatch.setattr(type(rt.ops), "_conv_walks", lambda *_: walks)
    ch, rows = 1024, 24
    z = -torch.linspace(20.0, 88.5, ch, device="cuda")
    zero = lambda *s: torch.zeros(s, dtype=dtype, device="cuda")
    got = rt.ops.causal_conv_silu(zero(rows, ch), zero(4, ch).float(), z, zero(1, 3, ch), context(rt, [0], [0], [rows], None).batch)
    silu = lambda t: t.double() * torch.sigmoid(t.double())
    unit = 1.01 * 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -21
    assert ((got.double() - silu(z)).abs() <= unit * silu(z).abs()).all()
    for rows in (24, 4096):  # a block a part, a warp a part
        y, gates, out = torch.ones((rows, ch), device="cuda"), z.to(dtype).repeat(rows, 1), zero(rows, ch)
        rt.ops.gated_group_norm(y, gates, torch.ones(ch, device="cuda"), 1, 1e-5, out, 0, 1.0)
        v = silu(gates)
        want = v / torch.sqrt((v * v).mean(-1, keepdim=True) + 1e-5)
        assert ((out.double() - want).abs() <= unit * want.abs()).all()


def test_a_tokens_infinities_reach_no_earlier_token_of_a_state_space_chunk(monkeypatch):
    rt = runtime(torch.bfloat16)
    monkeypatch.setattr(type(rt.ops), "SSD_TENSOR_MIN", 1)
    H, P, N = 2, 64, 32
    x, B, C = (rand((100, n), 40 + i).to(torch.bfloat16).cuda() for i, n in enumerate((H * P, N, N)))
    dt, vec = rand((100, H), 43).to(torch.bfloat16).cuda(), rand((H,), 44).cuda()
    ctx = context(rt, [0], [0], [100], None)
    got = []
    for value in (1.0, float("inf")):
        x = x.clone()
        x[41, 5] = value
        state = torch.zeros((1, H, N, P), device="cuda")
        got.append((rt.ops.ssd_scan(x, B, C, dt, vec, vec, vec, H, P, N, 1, state, ctx.batch), state))
    (y0, s0), (y1, s1) = got
    rest = [c for c in range(H * P) if c != 5]
    assert torch.equal(y0[:41], y1[:41]) and torch.equal(y0[:, rest], y1[:, rest]) and not torch.isfinite(y1[41:, 5]).any()
    assert torch.equal(s0[0, 1], s1[0, 1]) and not torch.isfinite(s1[0, 0, :, 5]).any()


def test_a_state_space_scan_without_room_for_its_scratch(monkeypatch):
    """Where the device's memory has no room for the chunks' states, a prompt goes through in smaller portions, and by the other
    scan where not even one chunk of each sequence fits."""
    rt = runtime(torch.bfloat16)
    H, P, N, lens = 4, 64, 128, [240, 70]  # shorter than the other scan's own chunks
    rows = sum(lens)
    x, B, C = (rand((rows, n), 40 + i).to(torch.bfloat16).cuda() for i, n in enumerate((H * P, N, N)))
    dt, vec = rand((rows, H), 43).to(torch.bfloat16).cuda(), rand((H,), 44).cuda()
    start = rand((2, H, N, P), 45).cuda()
    ctx = context(rt, [0, 1], [0, 0], lens, None)
    monkeypatch.setattr(type(rt.ops), "SSD_TENSOR_MIN", 1)
    empty, runs = torch.empty, {}
    item = 4 * 2 * H * N * P  # bytes of one chunk's states
    for name, room in (("all", 1 << 30), ("two chunks", 3 * item), ("none", item - 1)):
        def limited(*shape, room=room, **kw):
            n = math.prod(shape[0]) if isinstance(shape[0], (tuple, list)) else math.prod(shape)
            if kw.get("dtype") is torch.float32 and 4 * n > room and n != rows * H * P:  # the outputs are always there
                raise torch.OutOfMemoryError("no room")
            return empty(*shape, **kw)

        monkeypatch.setattr(torch, "empty", limited)
        state = start.clone()
        runs[name] = rt.ops.ssd_scan(x, B, C, dt, vec, vec, vec, H, P, N, 1, state, ctx.batch), state
        monkeypatch.setattr(torch, "empty", empty)
    monkeypatch.setattr(type(rt.ops), "SSD_TENSOR_MIN", 1 << 30)
    state = start.clone()
    runs["tokens"] = rt.ops.ssd_scan(x, B, C, dt, vec, vec, vec, H, P, N, 1, state, ctx.batch), state
    for a, b in (("two chunks", "all"), ("none", "tokens")):
        assert torch.equal(runs[a][0], runs[b][0]) and torch.equal(runs[a][1], runs[b][1]), a


def test_state_space_heads_that_forget_everything(monkeypatch):
    """Rates whose log decay is minus infinity in 32 bits (and so large that a sum of 64 bits would lose a later token's): a decay of
    zero, as the scan token by token has it, with step sizes that leave single tokens almost undecayed."""
    rt = runtime(torch.bfloat16)
    H, P, N, lens = 4, 64, 32, [150, 40]
    rows = sum(lens)
    x, B, C = (rand((rows, n), 40 + i).to(torch.bfloat16).cuda() for i, n in enumerate((H * P, N, N)))
    dt, vec = rand((rows, H), 43).to(torch.bfloat16).cuda(), rand((H,), 44).cuda()
    dt[::3] = -60.0
    bias, a_log = torch.zeros(H, device="cuda"), torch.tensor([100.0, 88.0, 57.0, 0.0], device="cuda")
    start = rand((2, H, N, P), 45).cuda()
    ctx = context(rt, [0, 1], [0, 0], lens, None)
    runs = []
    for least in (1, 1 << 30):
        monkeypatch.setattr(type(rt.ops), "SSD_TENSOR_MIN", least)
        state = start.clone()
        runs.append((rt.ops.ssd_scan(x, B, C, dt, bias, a_log, vec, H, P, N, 1, state, ctx.batch), state))
    for got, want in zip(*runs):
        assert torch.isfinite(want).all()
        assert ((got - want).double().norm() / want.double().norm()).item() < 2e-6


@pytest.mark.parametrize("dtype", DTYPES)
def test_a_state_carries_one_loud_token_over_hundreds(dtype):
    """A head whose decay is almost one keeps a token that came hundreds of tokens (and several chunks and
    steps) earlier; a state that were lost or reset at a chunk's or a step's edge would show as silence."""
    rt = runtime(dtype)
    shape = (32, 2, 16, 16, 1, 4, 1)
    part, m, ref = ssm_part(shape, dtype, rt)
    for t in (part.a_log, ref["A_log"]):
        t.fill_(-9.0)  # rate exp(-9): the state loses a tenth in a thousand tokens
    T, loud = 700, 5
    h = rand((T, 32), 3, 0.05)
    h[loud] *= 400.0
    h = h.to(dtype)
    want = plain.mamba2(h.double(), ref, "", m, 1e-5)
    quiet = h.clone()
    quiet[loud] = 0
    base = plain.mamba2(quiet.double(), ref, "", m, 1e-5)
    assert (want[600:] - base[600:]).abs().max() > 0.2 * want[600:].abs().max()  # the case shows what it is meant to
    for pieces in ([T], [300, 256, 144], [640] + [1] * 60):
        close(run_part(part, rt, h, pieces, dtype), want, dtype, f"far token, pieces {pieces[:3]}")


ATTN_SHAPES = [  # hidden, heads, kv_heads, dim, vdim, rot, base
    (72, 6, 3, 16, 16, 16, 1e4),
    (64, 4, 1, 32, 64, 8, 2e4),
    (40, 2, 2, 24, 8, 24, 50.0),
    (48, 3, 1, 8, 40, 2, 10.0),
    (50, 3, 3, 6, 5, 4, 7.0),
    (64, 4, 2, 32, 32, 0, 1e4),
]


def attention_part(shape, dtype, rt, seed=0, scale=0.4):
    from kernel_rush_kawk_b200.parts import SinkWindowAttention

    C, H, G, D, Dv, rot, base = shape
    m = {"heads": H, "kv_heads": G, "dim": D, "vdim": Dv, "scale": scale, "rot": {"dims": rot, "base": base}}
    part = SinkWindowAttention({"hidden": C, "heads": H, "kv_heads": G, "dim": D, "vdim": Dv, "scale": scale, "window": None,
                                "rot_dims": rot, "rot_base": base, "sink": "zero", "bias": True, "qk_norm": "row", "eps": 1e-5})
    w = {"q": rand((H * D, C), seed + 1, 0.4), "k": rand((G * D, C), seed + 2, 0.4), "v": rand((G * Dv, C), seed + 3, 0.3),
         "o": rand((C, H * Dv), seed + 4, 0.2), "q.b": rand((H * D,), seed + 5, 0.5), "k.b": rand((G * D,), seed + 6, 0.5),
         "v.b": rand((G * Dv,), seed + 7, 0.5), "q.norm": 1 + rand((H * D,), seed + 8, 0.3), "k.norm": 1 + rand((G * D,), seed + 9, 0.3)}
    assert {k: tuple(s.shape) for k, s in part.tensor_specs().items()} == {k: tuple(v.shape) for k, v in w.items()}
    dev, ref = as_path(w, dtype)
    part.bind(dev, rt)
    return part, m, ref


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("shape", ATTN_SHAPES)
def test_attention_with_biases_row_norms_and_the_zero_sink_alone(dtype, shape):
    rt = runtime(dtype)
    part, m, ref = attention_part(shape, dtype, rt)
    T = 200
    h = rand((T, shape[0]), 9).to(dtype)
    want = plain.attention(h.double(), ref, "", m, 1e-5)
    other = rand((80, shape[0]), 10).to(dtype)
    for pieces, prior in (([T], ()), ([63, 2, 64, 71], ()), ([150] + [1] * 50, ()), ([T], [(other, [80])])):
        close(run_part(part, rt, h, pieces, dtype, prior=prior), want, dtype, f"attention {shape}, pieces {pieces[:4]}")


@pytest.mark.parametrize("dtype", DTYPES)
def test_the_zero_sink_takes_its_share_and_the_first_token_is_not_alone(dtype):
    """With tiny scores every weight is 1 / (keys + 1): the first token's output is half its value, not all of it."""
    rt = runtime(dtype)
    shape = (32, 2, 1, 16, 16, 4, 100.0)
    part, m, ref = attention_part(shape, dtype, rt, scale=1e-6)
    m["scale"] = 1e-6
    part._w_out = torch.eye(32, dtype=dtype, device="cuda")
    ref["o"] = torch.eye(32, dtype=torch.float64)
    h = rand((20, 32), 3).to(dtype)
    got = run_part(part, rt, h, [20], dtype)
    close(got, plain.attention(h.double(), ref, "", m, 1e-5), dtype, "uniform weights with the sink's share")
    v = (h.double() @ ref["v"].T + ref["v.b"])
    close(got[:1, :16], v[:1] / 2, dtype, "the first token")
    close(got[9:10, :16], v[:10].sum(dim=0, keepdim=True) / 11, dtype, "the tenth token")


def far_key_case(loud, T, dtype):
    """Keys are made from the first query head's weights, and the loud token's input is three times the last
    token's: its key points the way of the last query (the row norm takes the factor out) while its value is its
    own, so the last row's output leans on that one key among hundreds."""
    shape = (32, 2, 1, 32, 32, 2, 1000.0)
    w_seed = 0
    C, H, G, D, Dv, rot, base = shape
    w = {"q": rand((H * D, C), w_seed + 1, 0.4), "v": rand((G * Dv, C), w_seed + 3, 0.3), "o": rand((C, H * Dv), w_seed + 4, 0.2),
         "q.b": rand((H * D,), w_seed + 5, 0.1), "v.b": rand((G * Dv,), w_seed + 7, 0.5), "q.norm": 1 + rand((H * D,), w_seed + 8, 0.1)}
    w.update({"k": w["q"][:D].clone(), "k.b": w["q.b"][:D].clone(), "k.norm": w["q.norm"][:D].clone()})
    h = rand((T, C), 21, 0.5)
    h[loud] = 3.0 * h[T - 1]
    return shape, w, h.to(dtype)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("loud, T", [(0, 70), (63, 200), (64, 200), (5, 600)])
def test_one_far_key_among_hundreds_is_found(dtype, loud, T):
    """The key of one token (the very first, at a page's edge, far back) stands out for the last query, in a
    whole prompt, decoded alone, and in pieces of two."""
    from kernel_rush_kawk_b200.parts import SinkWindowAttention

    rt = runtime(dtype)
    shape, w, h = far_key_case(loud, T, dtype)
    C, H, G, D, Dv, rot, base = shape
    m = {"heads": H, "kv_heads": G, "dim": D, "vdim": Dv, "scale": 0.7, "rot": {"dims": rot, "base": base}}
    part = SinkWindowAttention({"hidden": C, "heads": H, "kv_heads": G, "dim": D, "vdim": Dv, "scale": 0.7, "window": None,
                                "rot_dims": rot, "rot_base": base, "sink": "zero", "bias": True, "qk_norm": "row", "eps": 1e-5})
    dev, ref = as_path(w, dtype)
    part.bind(dev, rt)
    want = plain.attention(h.double(), ref, "", m, 1e-5)
    without = h.double().clone()
    without[loud] = rand((C,), 77, 0.5).double()
    other = plain.attention(without, ref, "", m, 1e-5)
    assert (want[-1] - other[-1]).abs().max() > 0.2 * want[-1].abs().max()  # the case shows what it is meant to
    for pieces in ([T], [T - 3, 1, 1, 1], [2] * (T // 2)):
        close(run_part(part, rt, h, pieces, dtype), want, dtype, f"loud token {loud} of {T}, pieces {pieces[:3]}")


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("rows, inter, limit, C", [(5, 24, 1.0, 48), (40, 33, 0.6, 48), (3, 64, 7.0, 48),
                                                   (5, 40, 1.0, 64), (13, 96, 0.8, 128), (1, 33, 0.5, 96)])
def test_dense_feed_forward_with_clamped_inputs(dtype, rows, inter, limit, C):
    """Widths that are a multiple of 32 take, for few bfloat16 rows, the product whose epilogue clamps and
    multiplies; the others the product and the activation kernel."""
    from kernel_rush_kawk_b200.parts import GatedMLP

    rt = runtime(dtype)
    part = GatedMLP({"hidden": C, "intermediate": inter, "activation": "swish_clamped", "limit": limit, "slope": 1.702})
    w = {"gate": rand((inter, C), 1, 0.4), "up": rand((inter, C), 2, 0.4), "down": rand((C, inter), 3, 0.3)}
    dev, ref = as_path(w, dtype)
    part.bind(dev, rt)
    h = rand((rows, C), 4, 1.5).to(dtype)
    g = h.double() @ ref["gate"].T
    assert (g > limit).any() and (g < -limit).any()  # both sides of the clamps are exercised
    ctx = SimpleNamespace(ops=rt.ops)
    close(part.forward(ctx, h.cuda()), plain.dense_ff(h.double(), ref, "", {"limit": limit}), dtype, "clamped dense feed-forward")


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("shape", [(64, 5, 2, 40), (96, 8, 1, 48), (50, 3, 3, 11), (64, 16, 4, 32), (32, 40, 5, 16)])
@pytest.mark.parametrize("rows", [1, 5, 200])
def test_experts_weighted_by_the_softmax_over_all_of_them(dtype, shape, rows):
    from kernel_rush_kawk_b200.parts import RoutedExperts

    rt = runtime(dtype)
    C, E, top, F = shape
    part = RoutedExperts({"hidden": C, "experts": E, "top": top, "intermediate": F, "router_bias": False, "weights": "all"})
    w = {"router": rand((E, C), 1, 0.5)}
    for e in range(E):
        w.update({f"e{e}.gate": rand((F, C), 10 + 3 * e, 0.3), f"e{e}.up": rand((F, C), 11 + 3 * e, 0.3),
                  f"e{e}.down": rand((C, F), 12 + 3 * e, 0.3)})
    assert {k: tuple(s.shape) for k, s in part.tensor_specs().items()} == {k: tuple(v.shape) for k, v in w.items()}
    dev, ref = as_path(w, dtype)
    part.bind(dev, rt)
    h = rand((rows, C), 7, 1.5).to(dtype)
    want = plain.routed_ff(h.double(), ref, "", {"router": {"experts": E, "top": top}})
    for decode in (False, True):
        ctx = SimpleNamespace(ops=rt.ops, batch=SimpleNamespace(is_decode=decode))
        close(part.forward(ctx, h.cuda()), want, dtype, f"experts {shape}, {rows} rows, single-token step {decode}")


def test_routing_weights_are_shares_of_the_whole_softmax():
    rt = runtime(torch.float32)
    x = torch.eye(4, device="cuda")
    w = torch.tensor([[1.0, 2.0, 0.0, -1.0], [3.0, 2.0, 0.0, 5.0], [3.0, 0.5, 0.0, 5.0], [0.0, 2.0, 0.0, 4.0]], device="cuda").t().contiguous()
    experts, weights, _ = rt.ops.moe_route(x, w, None, 2, over_all=True)
    z = x @ w.t()
    for r in range(4):
        best = sorted(range(4), key=lambda e: (-float(z[r, e]), e))[:2]
        assert experts[r].tolist() == best
        assert torch.allclose(weights[r], torch.softmax(z[r], dim=0)[best], atol=1e-6)
        assert float(weights[r].sum()) < 1.0


# ----------------------------------------------------------------------------------------------
# the model through the engine
# ----------------------------------------------------------------------------------------------

def engine(folder, dtype, **kw):
    from kernel_rush_kawk_b200 import Engine

    args = dict(dtype=dtype, max_tokens=4096, max_slots=6, max_context=1024)
    args.update(kw)
    return Engine(folder, **args)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("name", list(CONFIGS))
def test_whole_portions_and_single_tokens_through_the_engine(folders, name, dtype):
    from kernel_rush_kawk_b200 import StepEntry

    eng = engine(folders[name], dtype)
    ids = prompts(name, [300])[0]
    ref = plain_logits(folders[name], ids)
    for pieces in ([300], [130, 2, 3, 64, 101], [250] + [1] * 50):
        slot = eng.cache.alloc()
        got, start = [], 0
        for n in pieces:
            got.append(eng.step([StepEntry(slot, ids[start:start + n], list(range(n)))]).clone())
            start += n
        eng.cache.free(slot)
        assert_logits(torch.cat(got), ref, dtype, f"{name} {dtype}, pieces {pieces[:4]}")
    eng.cache.check()


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_unequal_batches_reused_slots_and_long_decoding(folders, dtype):
    """Five requests of unequal length start together (one long enough for the scan in chunks beside short ones)
    and are decoded together while the shorter ones end; their slots, states and pages are then used again by
    others. Every row against the sequence run alone in the plain implementation."""
    from kernel_rush_kawk_b200 import StepEntry

    name = "za"
    eng = engine(folders[name], dtype, max_slots=5)
    for round_ in range(2):
        lengths = [90, 1, 400, 37, 64] if round_ == 0 else [65, 130, 2]
        tails = [70, 0, 100, 20, 1] if round_ == 0 else [30, 60, 1]
        seqs = prompts(name, lengths, seed=5 + round_)
        slots = [eng.cache.alloc() for _ in seqs]
        heads = [len(ids) - t for ids, t in zip(seqs, tails)]
        first = eng.step([StepEntry(s, ids[:n], [n - 1]) for s, ids, n in zip(slots, seqs, heads)]).clone()
        for i, (ids, n) in enumerate(zip(seqs, heads)):
            assert_logits(first[i:i + 1], plain_logits(folders[name], ids)[n - 1:n], dtype, f"round {round_}, prompt {i}")
        got = {i: [] for i in range(len(seqs))}
        for t in range(max(tails)):
            live = [i for i in range(len(seqs)) if t < tails[i]]
            out = eng.step([StepEntry(slots[i], [seqs[i][heads[i] + t]], [0]) for i in live])
            for row, i in enumerate(live):
                got[i].append(out[row].clone())
            for i in range(len(seqs)):
                if t + 1 == tails[i]:
                    eng.cache.free(slots[i])
        for i, ids in enumerate(seqs):
            if tails[i] == 0:
                eng.cache.free(slots[i])
                continue
            assert_logits(torch.stack(got[i]), plain_logits(folders[name], ids)[heads[i]:], dtype, f"round {round_}, decoded sequence {i}")
        eng.cache.check()
        assert eng.cache.live == 0


def test_greedy_generation_through_the_engines_own_entry(folders):
    """Engine.generate (scheduler, captured single-token steps, selection kernel) against greedy decoding
    with the plain implementation; prompts of unequal length, one of a single token."""
    name = "zb"
    eng = engine(folders[name], "float32", max_tokens=None)
    seqs = prompts(name, [33, 1, 80], seed=9)
    steps = list(eng.generate(seqs, 12))
    assert len(steps) == 12
    cfg, w = plain.read_folder(folders[name], torch.float64)
    for i, ids in enumerate(seqs):
        ids = list(ids)
        for t in range(12):
            logits = plain.forward(cfg, w, ids)[-1]
            best = torch.topk(logits, 2).values
            if best[0] - best[1] < 1e-4:  # too close to call in 32-bit: stop comparing this sequence
                break
            assert steps[t][i] == int(logits.argmax()), f"sequence {i}, new token {t}"
            ids.append(steps[t][i])


def test_trace_replay_serves_the_design(folders, tmp_path):
    """bin/trace_run's program on a small schedule: a batch of prompts, single tokens, a request that ends."""
    from kernel_rush_kawk_b200 import replay

    name = "zc"
    a, b = prompts(name, [70, 9], seed=4)
    lines = [{"step": 0, "entries": [{"id": "a", "tokens": a[:60], "want": [0, 59]}, {"id": "b", "tokens": b[:8], "want": [7]}], "end": []},
             {"step": 1, "entries": [{"id": "a", "tokens": [a[60]], "want": [0]}, {"id": "b", "tokens": [b[8]], "want": []}], "end": ["b"]}]
    lines += [{"step": 2 + t, "entries": [{"id": "a", "tokens": [a[61 + t]], "want": [0]}], "end": ["a"] if t == 8 else []} for t in range(9)]
    out = io.StringIO()
    args = replay.build_parser().parse_args(["--model", str(folders[name]), "--dtype", "float32", "--out", str(tmp_path / "o"),
                                             "--max-tokens", "256"])
    assert replay.run(args, stdin=io.StringIO("\n".join(json.dumps(l) for l in lines) + "\n"), stdout=out) == 0
    assert out.getvalue().split() == [w for t in range(11) for w in ("done", str(t))]
    import numpy as np
    ref_a, ref_b = plain_logits(folders[name], a), plain_logits(folders[name], b)
    first = torch.from_numpy(np.fromfile(tmp_path / "o" / "0.f32", dtype="<f4").reshape(3, -1))
    assert_logits(first, torch.stack([ref_a[0], ref_a[59], ref_b[7]]), "float32", "replayed prompts")
    for t in range(10):
        row = torch.from_numpy(np.fromfile(tmp_path / "o" / f"{1 + t}.f32", dtype="<f4").reshape(1, -1))
        assert_logits(row, ref_a[60 + t:61 + t], "float32", f"replayed token {t}")
