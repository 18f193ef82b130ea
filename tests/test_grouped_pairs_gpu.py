"""The grouped products of the routed experts at the edges of their tiles: rows of an expert around multiples of 32 and 256,
more experts than a warp has lanes, empty ones, and widths at which the second block of a pair has part of a tile or nothing."""

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


@pytest.mark.parametrize("E, top, F, C, line", [(64, 6, 640, 1280, 24), (8, 2, 96, 72, 48)])
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
