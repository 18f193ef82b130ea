"""The kernels' error word on the serving path: a bounded wait that runs out, a bad id that reaches
the device, and what generation does about them. Nothing here faults or hangs the device: the
waiting kernel gives up after a millisecond on a barrier that nobody arrives at, and the gather
kernel bounds-checks the id, writes zeros and sets the word."""

import pytest
import torch

from helpers import prompts_for

pytestmark = pytest.mark.gpu


def engine_of(folders, name="tiny_a", **kw):
    from kernel_rush_kawk_b200 import Engine

    return Engine(folders[name], dtype="bfloat16", max_slots=4, **kw)


def test_a_wait_that_runs_out_sets_the_word_and_check_raises(folders):
    from kernel_rush_kawk_b200.csrc import KernelError

    engine = engine_of(folders)
    ops = engine.ops
    ops.check()
    ops.selftest_wait_runs_out(limit_us=1000)
    with pytest.raises(KernelError, match="ran out"):
        ops.check()
    ops.check()  # the word was cleared: the context is as usable as before
    assert len(list(engine.generate(prompts_for("tiny_a", [5]), 3))) == 3


def test_generate_raises_on_a_flag_and_the_next_request_is_right(folders):
    from kernel_rush_kawk_b200.csrc import KernelError

    engine = engine_of(folders)
    prompts = prompts_for("tiny_a", [9, 4], seed=41)
    want = list(engine.generate(prompts, 10))
    # a token id beyond the table reaches the gather kernel directly: it writes a zero row and sets the word
    bad = torch.tensor([5, 100000], dtype=torch.int32, device="cuda")
    rows = engine.ops.embed(engine.model.embedding.table, bad, 2)
    torch.cuda.synchronize()
    assert rows[1].abs().max().item() == 0
    with pytest.raises(KernelError, match="token id"):
        list(engine.generate(prompts, 10))
    assert engine.cache.live == 0, "the failed call gave its slots back"
    engine.cache.check()
    assert list(engine.generate(prompts, 10)) == want, "the flag is cleared by the raise; the next request is served"


def test_a_flag_raised_while_steps_run_ahead_surfaces_with_their_tokens(folders):
    from kernel_rush_kawk_b200.csrc import KernelError

    engine = engine_of(folders)
    prompts = prompts_for("tiny_a", [7, 3], seed=42)
    it = engine.generate(prompts, 12)
    next(it)
    next(it)
    engine.ops.selftest_wait_runs_out(limit_us=500)  # lands between queued steps
    with pytest.raises(KernelError):
        for _ in it:
            pass
    assert engine.cache.live == 0
    assert len(list(engine.generate(prompts, 4))) == 4


def test_a_multi_token_step_ends_with_a_look_at_the_word(folders):
    from kernel_rush_kawk_b200 import StepEntry
    from kernel_rush_kawk_b200.csrc import KernelError

    engine = engine_of(folders, max_tokens=1024)
    slot = engine.cache.alloc()
    engine.ops.selftest_wait_runs_out(limit_us=500)
    with pytest.raises(KernelError):
        engine.step([StepEntry(slot, [1, 2, 3], [2])])
    engine.cache.free(slot)
    slot = engine.cache.alloc()
    assert engine.step([StepEntry(slot, [1, 2, 3], [2])]).shape[0] == 1
    engine.cache.free(slot)


def test_rebuilding_the_cache_gives_its_memory_back(folders):
    """Without a fixed ``max_tokens`` the cache is rebuilt when a call needs more room; the old storage
    must go (no part of the engine may keep the old cache alive)."""
    engine = engine_of(folders)
    list(engine.generate(prompts_for("tiny_a", [5]), 2))
    torch.cuda.synchronize()
    sizes = []
    for n in (400, 900, 1500):
        list(engine.generate(prompts_for("tiny_a", [n]), 2))
        torch.cuda.synchronize()
        sizes.append((engine.cache.bytes(), torch.cuda.memory_allocated()))
    growth_cache = sizes[-1][0] - sizes[0][0]
    growth_alloc = sizes[-1][1] - sizes[0][1]
    assert growth_alloc <= growth_cache + (8 << 20), f"allocated memory grew by {growth_alloc}, the cache itself by {growth_cache}"


@pytest.mark.parametrize("depth,asked", [(2, 0), (2, 1), (2, 2), (2, 3), (3, 2), (3, 7), (3, 9), (6, 5), (6, 13), (8, 64)])
def test_a_block_that_gives_up_waits_for_the_copies_that_it_asked_for(folders, depth, asked):
    """What a kernel with a ring of copies calls before it ends early: every slice asked for and read by nobody is in shared memory
    afterwards, from a ring that is not full to one that has gone round, and a copy that never comes costs its limit and no more."""
    from kernel_rush_kawk_b200.csrc import KernelError

    ops = engine_of(folders).ops
    ops.check()
    src = torch.randn(64 * 256, device="cuda")
    want = torch.zeros((depth, 256), device="cuda")
    for i in range(asked):
        want[i % depth] = src[i * 256:(i + 1) * 256]
    assert torch.equal(ops.selftest_wait_for_copies(src, depth, asked), want)
    ops.check()
    assert torch.equal(ops.selftest_wait_for_copies(src, depth, asked, withheld=1), want)
    with pytest.raises(KernelError, match="ran out"):
        ops.check()
    ops.check()


@pytest.mark.parametrize("rows", [130, 700])
def test_attention_blocks_that_find_a_give_up_code_leave_and_the_next_kernels_are_right(rows):
    """Blocks of the prompt attention that find a code of an earlier kernel in the error word have asked for their query tiles already: they
    wait for those, write nothing and leave, launch after launch, and what runs right behind them on the same SMs (products with
    rings of copies and barriers of their own, then the same attention) gives its usual bits."""
    from test_kernels_gpu import make_batch, make_cache, rand

    from kernel_rush_kawk_b200.csrc import KernelError, load_kernels

    ops = load_kernels((128,), "cuda:0")
    heads, kv_heads, D = 32, 8, 128
    cache = make_cache(24, kv_heads, D, 1, 20, torch.bfloat16, 90)
    batch = make_batch([0], [300], [rows])
    qkv = rand((rows, (heads + 2 * kv_heads) * D), torch.bfloat16, 91)
    ops.qk_norm_rope_write(qkv, heads, kv_heads, D, None, None, 1e-6, None, None, batch, cache)
    x, w = rand((8, 1024), torch.float32, 92), rand((4096, 1024), torch.float32, 93)
    attend = lambda out: ops.attn[D].krk_attention_prefill_tcgen05(
        out.data_ptr(), qkv.data_ptr(), qkv.stride(0), heads, kv_heads, batch.seq_slot.data_ptr(), batch.seq_start.data_ptr(),
        batch.seq_qlen.data_ptr(), batch.cu_q.data_ptr(), cache.table.data_ptr(), cache.width, cache.k.data_ptr(), cache.v.data_ptr(),
        cache.k.shape[0], 1, rows, rows, D ** -0.5, 0, ops.error.data_ptr(), ops._stream())
    out = torch.zeros((rows, heads * D), dtype=torch.bfloat16, device="cuda")
    assert attend(out) == 0
    want = out.clone(), ops.linear(x, w)
    ops.check()
    for _ in range(20):
        out.fill_(7.0)
        ops.error.fill_(8)
        assert attend(out) == 0
        got = ops.linear(x, w)
        assert torch.equal(out, torch.full_like(out, 7.0)) and torch.equal(got, want[1])
        with pytest.raises(KernelError, match="barrier wait"):
            ops.check()
        assert attend(out) == 0
        ops.check()
        assert torch.equal(out, want[0])
