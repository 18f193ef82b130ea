"""The grouped products of the routed experts at the edges of their tiles: rows of an expert around multiples of 32 and 256,
more experts than a warp has lanes, empty ones, and widths at which the second block of a pair has part of a tile or nothing; by pairs of
blocks, by single ones and in a single-token step's small tiles."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gated", [0, 1])
@pytest.mark.parametrize("N, K, counts", [
    (8, 64, [31, 32, 33, 0, 1]),
    (72, 88, [255, 256, 257, 0, 63, 65]),
    (136, 200, [511, 513, 0, 0, 769]),
    (248, 72, [17 * (e % 4 == 0) + e % 3 for e in range(70)]),
    (264, 640, [2049, 5]),
    (384, 136, [0] * 40 + [1] + [0] * 30 + [300]),
])
def test_tiles_of_an_experts_rows_at_their_edges(N, K, counts, gated):
    from kernel_rush_kawk_b200.csrc import load_kernels

    ops = load_kernels((), "cuda:0")
    g = torch.Generator().manual_seed(1)
    rand = lambda *shape: torch.randn(shape, generator=g)
    E = len(counts)
    offsets = torch.tensor([0] + counts).cumsum(0).to(torch.int32)
    rows = int(offsets[-1])
    a, w = rand(rows + 3, K).to(torch.bfloat16), (rand(E, (2 if gated else 1) * N, K) * K ** -0.5).to(torch.bfloat16)
    a_d, w_d, o_d = a.cuda(), w.cuda(), offsets.cuda()
    for tall in (0, 1):
        out = torch.full((rows + 3, N), 7.0, dtype=torch.bfloat16, device="cuda")
        ops._ok(ops.moe.krk_grouped_gemm(out.data_ptr(), a_d.data_ptr(), w_d.data_ptr(), o_d.data_ptr(), rows + 3, E, N, K,
                                         0 if gated else -1, gated, tall, None, 0.0, 0.0, ops.error.data_ptr(), ops._stream()),
                "grouped product")
        want = torch.full((rows + 3, N), 7.0, dtype=torch.float64)  # rows beyond the last expert's stay as they were
        bound = torch.zeros_like(want)
        for e in range(E):
            lo, hi = int(offsets[e]), int(offsets[e + 1])
            y = a[lo:hi].double() @ w[e].double().t()
            if gated:
                # rounding to bfloat16 moves gate, up and result by up to 2^-8 of themselves, the gate's through silu's slope
                gate, up, s = y[:, :N], y[:, N:], torch.sigmoid(y[:, :N])
                want[lo:hi] = gate * s * up
                bound[lo:hi] = 2.0 ** -8 * ((gate * (s + gate * s * (1 - s)) * up).abs() + 2 * want[lo:hi].abs())
            else:
                want[lo:hi] = y
                bound[lo:hi] = 2.0 ** -8 * y.abs()
        # float32 sums of up to 640 products of order K^-1/2, and the next order of the roundings
        assert bool(((out.double().cpu() - want).abs() <= 1.02 * bound + 1e-4).all()), f"tall {tall}"
    ops.check()


@pytest.mark.parametrize("E, top, F, C, line", [(64, 6, 640, 1280, 96), (8, 2, 96, 72, 48)])
def test_experts_where_their_products_change_hands(E, top, F, C, line):
    """Single-token steps and prompts of as many rows as move the experts' products from a block per piece of an expert to the grouped
    launches, and one row fewer and more: the same sums, within the roundings of each expert's two products."""
    from types import SimpleNamespace

    from kernel_rush_kawk_b200.csrc import load_kernels

    ops = load_kernels((), "cuda:0")
    assert ops._grouped_from(E, F, C, True) == line * top
    g = torch.Generator().manual_seed(2)
    K = 64
    w1 = (torch.randn(E, 2 * F, K, generator=g) * K ** -0.5).to(torch.bfloat16)
    w2 = (torch.randn(E, C, F, generator=g) * F ** -0.5).to(torch.bfloat16)
    for rows in (line - 1, line, line + 1):
        x = torch.randn(rows, K, generator=g).to(torch.bfloat16)
        experts = torch.stack([torch.randperm(E, generator=g)[:top] for _ in range(rows)]).int()
        weights = torch.rand(rows, top, generator=g)
        want = torch.zeros(rows, C, dtype=torch.float64)
        for r in range(rows):
            for j in range(top):
                e = int(experts[r, j])
                y = w1[e].double() @ x[r].double()
                want[r] += weights[r, j].double() * (w2[e].double() @ (y[:F] * torch.sigmoid(y[:F]) * y[F:]))
        for decode in (False, True):
            got = ops.moe_experts(x.cuda(), w1.cuda(), w2.cuda(), experts.cuda(), weights.cuda(), F, "silu",
                                  batch=SimpleNamespace(is_decode=decode))
            off = (got.double().cpu() - want).norm() / want.norm()
            # gate, up, their product, each expert's result and the sum are rounded: five times 2^-9 in the mean, added in squares
            assert off < 5 ** 0.5 * 2.0 ** -8, (rows, decode, float(off))
    ops.check()


@pytest.mark.parametrize("activation, act_params, weigh_input", [("silu", None, False), ("swish_clamped", (7.0, 1.702), True)])
def test_single_token_steps_are_as_exact_by_either_route(activation, act_params, weigh_input, monkeypatch):
    """Outputs next to the correctly rounded ones, where every product, activation and result is rounded as the path rounds it: by pieces of an
    expert half a percent or less, and no more by the grouped launches (4 % with one accumulator for all of k, whose last bits the
    tensor cores cut off)."""
    from types import SimpleNamespace

    from kernel_rush_kawk_b200.csrc import load_kernels
    from kernel_rush_kawk_b200.csrc.bindings import Kernels

    ops = load_kernels((), "cuda:0")
    g = torch.Generator("cuda").manual_seed(3)
    E, top, F, K, C, rows = 64, 6, 640, 2048, 1280, 64
    normal = lambda *s, std=1.0: torch.empty(s, device="cuda").normal_(0, std, generator=g)
    x, w1, w2 = (t.to(torch.bfloat16) for t in (normal(rows, K), normal(E, 2 * F, K, std=K ** -0.5), normal(E, C, F, std=F ** -0.5)))
    experts = torch.rand((rows, E), device="cuda", generator=g).topk(top, 1).indices.int()
    weights = torch.rand((rows, top), device="cuda", generator=g)
    rounded = lambda t: t.float().to(torch.bfloat16).double()
    want = torch.zeros((rows, C), dtype=torch.float64, device="cuda")
    for e in range(E):
        r, j = (experts == e).nonzero(as_tuple=True)
        y, w = x[r].double() @ w1[e].double().t(), weights[r, j].double()[:, None]
        if activation == "silu":
            y = rounded(y)
            h = y[:, :F] * torch.sigmoid(y[:, :F]) * y[:, F:]
        else:
            gate, up = (w * y)[:, :F].clamp(max=7.0), (w * y)[:, F:].clamp(-7.0, 7.0)
            h = gate * torch.sigmoid(1.702 * gate) * (up + 1)
        out = rounded(rounded(h) @ w2[e].double().t())
        want.index_add_(0, r, out if weigh_input else out * w)
    share = {}
    for route, line in (("pieces", 1 << 30), ("grouped", 0)):
        monkeypatch.setattr(Kernels, "_grouped_from", staticmethod(lambda *_, line=line: line))
        got = ops.moe_experts(x, w1, w2, experts, weights, F, activation, batch=SimpleNamespace(is_decode=True), act_params=act_params,
                              weigh_input=weigh_input)
        share[route] = (got != want.float().to(torch.bfloat16)).double().mean().item()
    ops.check()
    assert share["grouped"] < 1.5 * share["pieces"] + 1e-3 and share["pieces"] < 0.01, share


def test_gates_of_the_most_negative_in_a_single_token_step():
    """Gates down to where e^-g still is a number: activations of 1e-36 as exact as any other."""
    from kernel_rush_kawk_b200.csrc import load_kernels

    ops = load_kernels((), "cuda:0")
    N, K = 128, 64
    z = -torch.linspace(20.0, 87.5, N).to(torch.bfloat16)
    w = torch.zeros(1, 2 * N, K, dtype=torch.bfloat16)
    w[0, :N, 0], w[0, N:, 1] = z, 1.0
    a = torch.zeros(7, K, dtype=torch.bfloat16)
    a[:, :2] = 1.0
    out, offsets = torch.empty(7, N, dtype=torch.bfloat16, device="cuda"), torch.tensor([0, 7], dtype=torch.int32, device="cuda")
    a_d, w_d = a.cuda(), w.cuda()
    ops._ok(ops.moe.krk_grouped_gemm(out.data_ptr(), a_d.data_ptr(), w_d.data_ptr(), offsets.data_ptr(), 7, 1, N, K, 0, 1, 2, None, 0.0, 0.0,
                                     ops.error.data_ptr(), ops._stream()), "grouped product")
    want = z.double() * torch.sigmoid(z.double())
    assert ((out.double().cpu() - want).abs() <= 1.01 * 2.0 ** -8 * want.abs()).all()


@pytest.mark.parametrize("gated", [0, 1])
@pytest.mark.parametrize("N, K, counts", [(8, 64, [31, 32, 33, 0, 1]), (136, 200, [65, 0, 0, 97]), (264, 640, [2, 5]), (384, 520, [0] * 40 + [1] + [0] * 30 + [300])])
def test_single_token_tiles_at_their_edges(N, K, counts, gated):
    """Tiles of 32 rows in up to eight partial sums, fewer where k has fewer blocks of 64: within the rounding of the result and of a
    float32 sum, rows beyond the last expert's as they were."""
    from kernel_rush_kawk_b200.csrc import load_kernels

    ops = load_kernels((), "cuda:0")
    g = torch.Generator().manual_seed(4)
    offsets = torch.tensor([0] + counts).cumsum(0).to(torch.int32)
    rows, E = int(offsets[-1]), len(counts)
    a = torch.randn(rows + 3, K, generator=g).to(torch.bfloat16)
    w = (torch.randn(E, (2 if gated else 1) * N, K, generator=g) * K ** -0.5).to(torch.bfloat16)
    a_d, w_d, o_d = a.cuda(), w.cuda(), offsets.cuda()
    outs = []
    for tiles in (1, 2):
        out = torch.full((rows + 3, N), 7.0, dtype=torch.bfloat16, device="cuda")
        ops._ok(ops.moe.krk_grouped_gemm(out.data_ptr(), a_d.data_ptr(), w_d.data_ptr(), o_d.data_ptr(), rows + 3, E, N, K,
                                         0 if gated else -1, gated, tiles, None, 0.0, 0.0, ops.error.data_ptr(), ops._stream()), "grouped product")
        outs.append(out.double().cpu())
    ops.check()
    # one rounding of the result, gated of either product too (a gate's through silu's slope, at most 1.1)
    assert ((outs[0] - outs[1]).abs() <= (3.1 if gated else 1.0) * 2.0 ** -7 * outs[0].abs() + (2.0 ** -7 if gated else 1e-4)).all()
    assert (outs[1][rows:] == 7.0).all()


@pytest.mark.parametrize("gated, act", [(0, -1), (0, 5), (1, 0), (1, 3)])
@pytest.mark.parametrize("E, N, K, rows", [(8, 512, 128, 4100), (40, 128, 72, 500), (40, 72, 200, 3000), (8, 328, 640, 900), (4, 1032, 136, 2100)])
def test_single_blocks_and_pairs_are_the_same_bits(E, N, K, rows, gated, act):
    """Products of few tiles take single blocks (of these all plain ones, of the gated ones the first and the last): the same bits as by
    pairs, row weights and an expert without rows among them."""
    from kernel_rush_kawk_b200.csrc import load_kernels

    ops = load_kernels((), "cuda:0")
    g = torch.Generator().manual_seed(7)
    counts = torch.bincount(torch.randint(0, E - 1, (rows,), generator=g), minlength=E)
    offsets = torch.cat([torch.zeros(1, dtype=torch.long), counts.cumsum(0)]).int().cuda()
    a = torch.randn(rows, K, generator=g).to(torch.bfloat16).cuda()
    w = (torch.randn(E, (2 if gated else 1) * N, K, generator=g) * K ** -0.5).to(torch.bfloat16).cuda()
    weights = torch.rand(rows, generator=g).cuda() if act == 3 else None
    outs = []
    for route in (0, 1):
        out = torch.full((rows, N), 7.0, dtype=torch.bfloat16, device="cuda")
        ops._ok(ops.moe.krk_grouped_gemm(out.data_ptr(), a.data_ptr(), w.data_ptr(), offsets.data_ptr(), rows, E, N, K, act, gated, route,
                                         None if weights is None else weights.data_ptr(), 7.0, 1.702, ops.error.data_ptr(), ops._stream()),
                "grouped product")
        outs.append(out)
    ops.check()
    assert torch.equal(*outs)


@pytest.mark.parametrize("top, C", [(1, 64), (3, 72), (8, 2056), (11, 128)])
def test_the_sum_of_many_rows_is_that_of_few(top, C):
    """A row's chosen results added four or eight at a time: the same bits in a step of 445 rows as in one of 444, in the order of the choice."""
    from kernel_rush_kawk_b200.csrc import load_kernels

    ops = load_kernels((), "cuda:0")
    g = torch.Generator().manual_seed(8)
    rows, E = 445, 16
    x, yg = torch.randn(rows, C, generator=g).to(torch.bfloat16), torch.randn(rows * top, C, generator=g).to(torch.bfloat16)
    experts = torch.stack([torch.randperm(E, generator=g)[:top] for _ in range(rows)]).int()
    experts[torch.rand(rows, top, generator=g) < 0.1] = -1
    weights, passed = torch.rand(rows, top, generator=g), torch.rand(rows, generator=g)
    want = passed[:, None].double() * x.double()
    for j in range(top):
        want += torch.where(experts[:, j] < 0, 0.0, weights[:, j])[:, None].double() * yg.view(rows, top, C)[:, j].double()
    x_d, y_d, e_d, w_d, p_d = x.cuda(), yg.cuda(), experts.cuda(), weights.cuda(), passed.cuda()
    outs = []
    for n in (rows, rows - 1):
        out = torch.empty((rows, C), dtype=torch.bfloat16, device="cuda")
        ops._ok(ops.moe.krk_moe_combine(out.data_ptr(), None, None, y_d.data_ptr(), None, e_d.data_ptr(), None, 0, w_d.data_ptr(), n, top, C,
                                        x_d.data_ptr(), C, p_d.data_ptr(), 1, ops._stream()), "experts' sum")
        outs.append(out[:rows - 1])
    assert torch.equal(*outs)
    # one rounding to bfloat16, and float32 sums of up to twelve products of order one
    assert ((outs[0].double().cpu() - want[:-1]).abs() <= 1.01 * 2.0 ** -8 * want[:-1].abs() + 1e-5).all()


def test_single_token_steps_of_more_pairs_than_a_piece_holds(monkeypatch):
    """From 4,097 pairs on the kernel that reads an expert's weights once for its rows is out of bounds; the grouped launches, which take
    steps of fewer pairs, take those too, and the sums are as near 64 bits as by pairs, each of which reads its expert's weights itself."""
    from types import SimpleNamespace

    from kernel_rush_kawk_b200.csrc import load_kernels

    ops = load_kernels((), "cuda:0")
    g = torch.Generator().manual_seed(9)
    E, top, F, K, C = 32, 6, 96, 128, 72
    w1, w2 = (torch.randn(E, 2 * F, K, generator=g) * K ** -0.5).to(torch.bfloat16), (torch.randn(E, C, F, generator=g) * F ** -0.5).to(torch.bfloat16)
    grouped = []
    gemm = ops._grouped_experts
    monkeypatch.setattr(ops, "_grouped_experts", lambda *a: grouped.append(a[-1]) or gemm(*a))
    for rows in (682, 683):  # 4,092 and 4,098 pairs
        x = torch.randn(rows, K, generator=g).to(torch.bfloat16)
        experts = torch.stack([torch.randperm(E, generator=g)[:top] for _ in range(rows)]).int()
        weights = torch.rand(rows, top, generator=g)
        y = torch.einsum("rk,enk->ren", x.double(), w1.double())
        h = y[..., :F] * torch.sigmoid(y[..., :F]) * y[..., F:]
        each = torch.einsum("ref,ecf->rec", h, w2.double())
        want = (each.gather(1, experts.long()[..., None].expand(-1, -1, C)) * weights.double()[..., None]).sum(1)
        got = ops.moe_experts(x.cuda(), w1.cuda(), w2.cuda(), experts.cuda(), weights.cuda(), F, "silu", batch=SimpleNamespace(is_decode=True))
        off = (got.double().cpu() - want).norm() / want.norm()
        # gate, up, their product, each expert's result and the sum are rounded: five times 2^-9 in the mean, added in squares
        assert off < 5 ** 0.5 * 2.0 ** -8, (rows, float(off))
    ops.check()
    assert grouped == [2, 2], "both by the grouped launches, in a single-token step's tiles"


def test_a_captured_step_of_the_grouped_experts():
    """A single-token step by the grouped launches, captured and replayed over other rows, choices and weights: what the direct call returns."""
    from types import SimpleNamespace

    from kernel_rush_kawk_b200.csrc import load_kernels

    ops = load_kernels((), "cuda:0")
    g = torch.Generator().manual_seed(10)
    E, top, F, K, C, rows = 64, 6, 640, 128, 1280, 100
    w1, w2 = ((torch.randn(s, generator=g) * 0.06).to(torch.bfloat16).cuda() for s in ((E, 2 * F, K), (E, C, F)))

    def inputs():
        return (torch.randn(rows, K, generator=g).to(torch.bfloat16).cuda(),
                torch.stack([torch.randperm(E, generator=g)[:top] for _ in range(rows)]).int().cuda(), torch.rand(rows, top, generator=g).cuda())

    step = lambda x, experts, weights: ops.moe_experts(x, w1, w2, experts, weights, F, "silu", batch=SimpleNamespace(is_decode=True))
    assert rows * top >= ops._grouped_from(E, F, C, True)
    held = inputs()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        step(*held)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = step(*held)
    for _ in range(3):
        fresh = inputs()
        for a, b in zip(held, fresh):
            a.copy_(b)
        graph.replay()
        assert torch.equal(out, step(*fresh))
    ops.check()
