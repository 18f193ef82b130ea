"""Head norms and cache writes of bfloat16 steps of many rows, which take a block a row, and of fewer, which take a warp a head: within
roundings of 64 bits; the same bits however a prompt was cut; more heads than lanes take at once, odd counts of them, one and many sequences."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H, G, D", [(5, 1, 8), (3, 3, 16), (16, 4, 128), (40, 8, 128), (7, 2, 64), (9, 3, 256)])
@pytest.mark.parametrize("gains, temp", [(True, (0.1, 64)), (False, None)])
def test_rows_of_many_and_fewer(H, G, D, gains, temp):
    from kernel_rush_kawk_b200.cache.store import KVNeed, SequenceCache
    from kernel_rush_kawk_b200.csrc import load_kernels
    from kernel_rush_kawk_b200.engine import BatchMeta, StepContext

    ops, device = load_kernels((), "cuda:0"), torch.device("cuda:0")
    g = torch.Generator().manual_seed(5)
    n, eps = (H + 2 * G) * D, 1e-6
    proj = torch.randn(301, n + 16, generator=g).to(torch.bfloat16)
    gain = 1 + 0.2 * torch.randn(2 * D, generator=g)
    for lens, starts in (([256], [0]), ([255], [0]), ([300], [77]), ([100, 1, 190], [0, 700, 63])):
        rows = sum(lens)
        cache = SequenceCache([KVNeed(G, D)], 4096, len(lens), 2048, device, torch.bfloat16)
        slots = [cache.alloc() for _ in lens]
        for s, a, b in zip(slots, lens, starts):
            cache.reserve(s, a + b)
        cache.sync()
        meta = BatchMeta(rows, len(lens), 0, device)
        meta.fill(slots, starts, [[0] * a for a in lens], [])
        view = cache.view(0)
        x = proj[:rows].cuda()
        ops.bias_norm_rotate_write(x, 0, H * D, (H + G) * D, H, G, D, D, None, gain.cuda() if gains else None, eps,
                                   torch.zeros(0, device="cuda"), 0, False, StepContext(ops, meta, cache).batch, view, temperature=temp)
        at = torch.cat([torch.arange(b, b + a) for a, b in zip(lens, starts)])
        page = torch.cat([view.table[s].cpu().long()[torch.arange(b, b + a) // 64] for s, a, b in zip(slots, lens, starts)])
        want = proj[:rows, :n].double().view(rows, H + 2 * G, D)
        if gains:
            unit = want / (want.pow(2).mean(-1, keepdim=True) + eps).sqrt()
            want = torch.cat([unit[:, :H] * gain[:D].double(), unit[:, H:H + G] * gain[D:].double(), want[:, H + G:]], 1)
        if temp:
            want = want.clone()
            want[:, :H] *= (1 + temp[0] * torch.log(torch.floor((at.double() + 1) / temp[1]) + 1))[:, None, None]
        got = torch.cat([x.cpu()[:, :H * D].view(rows, H, D), view.k.cpu()[page, :, at % 64], view.v.cpu()[page, :, at % 64]], 1)
        assert ((got.double() - want).abs() <= 1.01 * 2.0 ** -8 * want.abs() + 1e-6).all(), (lens, starts)  # one rounding to bfloat16
        assert torch.equal(x.cpu()[:, H * D:], proj[:rows, H * D:]), "keys, values and what is behind them stay as they were"


@pytest.mark.parametrize("H, G, D", [(5, 1, 8), (3, 3, 16), (7, 2, 32), (7, 2, 64), (16, 4, 128), (40, 8, 128), (9, 3, 256)])
def test_portions_of_a_prompt_leave_the_same_bits(H, G, D):
    """A prompt whole (a block a row) and in portions (a warp a head): queries, keys and values do not depend on how it was cut."""
    from kernel_rush_kawk_b200.cache.store import KVNeed, SequenceCache
    from kernel_rush_kawk_b200.csrc import load_kernels
    from kernel_rush_kawk_b200.engine import BatchMeta, StepContext

    ops, device = load_kernels((), "cuda:0"), torch.device("cuda:0")
    g = torch.Generator().manual_seed(6)
    rows, n = 1500, (H + 2 * G) * D
    proj = torch.randn(rows, n, generator=g).to(torch.bfloat16).cuda()
    gain = (1 + 0.2 * torch.randn(2 * D, generator=g)).cuda()
    runs = []
    for lens in ([rows], [200] * 7 + [100]):
        cache = SequenceCache([KVNeed(G, D)], 2048, 1, 2048, device, torch.bfloat16)
        slot, x, at = cache.alloc(), proj.clone(), 0
        cache.reserve(slot, rows)
        cache.sync()
        view = cache.view(0)
        for some in lens:
            meta = BatchMeta(some, 1, 0, device)
            meta.fill([slot], [at], [[0] * some], [])
            ops.bias_norm_rotate_write(x[at:at + some], 0, H * D, (H + G) * D, H, G, D, D, None, gain, 1e-6, torch.zeros(0, device="cuda"), 0,
                                       False, StepContext(ops, meta, cache).batch, view, temperature=(0.1, 64))
            at += some
        pages = view.table[slot].cpu().long()[torch.arange(rows) // 64]
        runs.append((x.cpu(), view.k.cpu()[pages, :, torch.arange(rows) % 64], view.v.cpu()[pages, :, torch.arange(rows) % 64]))
    assert all(torch.equal(a, b) for a, b in zip(*runs))
