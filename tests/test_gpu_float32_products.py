"""The 32-bit products of larger matrices on tensor cores (`csrc/gemm_f32_split.cu`): no bit of a number is lost, whatever its
neighbours are, and no result is further from 64 bits than the multiply-adds (`csrc/gemm_f32.cu`) are."""
import numpy as np
import pytest
import torch

import ghost_infer_b200 as gi
from ghost_infer_b200.kernels import ops
from gpu_helpers import make_engine, tokens_for

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def plain(a, w):
    """The product by multiply-adds."""
    out, lib = torch.empty((a.shape[0], w.shape[0]), device=DEV), ops._bind()
    assert lib.gi_gemm_generic(out.data_ptr(), 0, ops.GEMM_STORE, a.data_ptr(), 0, w.data_ptr(), 0, a.shape[0], w.shape[0], a.shape[1],
                               a.stride(0), w.stride(0), out.stride(0), ops._stream()) == 0
    return out


def bound(a, w):
    """A number is three 16-bit floats with nothing left over.  Of sum |a w|: 1.01 * 2^-24 for the three small products that are left
    out; two instructions on a fresh accumulator, and an eighth of K's on one that holds at most 2^-6 of the whole (five
    products of 16 numbers each), which cut off 2^-23 at most; an addition for each 32 numbers, stretch and end."""
    chunks = (a.shape[1] + 63) // 64
    per = (chunks + 7) // 8
    return (a.double().abs() @ w.double().abs().T) * (1.01 * 2.0 ** -24 + (2 + 20 * per * 2.0 ** -6) * 2.0 ** -23 + (2 * per + 10) * 2.0 ** -24)


@pytest.mark.parametrize("m", [5, 70])
@pytest.mark.parametrize("spread", [8, 12, 16, 20, 40])
def test_neighbours_of_very_different_size(m, spread):
    """Channels scaled by 2^e, their weights by 2^-e: every product counts alike."""
    n, k, g = 1024, 1100, gen(spread)
    e = torch.randint(-spread, spread + 1, (k,), generator=g, device=DEV).float()
    a = torch.randn((m, k), generator=g, device=DEV) * torch.exp2(e)
    w = torch.randn((n, k), generator=g, device=DEV) * torch.exp2(-e)
    assert ((ops.gemm_generic(a, w).double() - a.double() @ w.double().T).abs() <= bound(a, w)).all()


@pytest.mark.parametrize("m", [5, 70])
@pytest.mark.parametrize("size", [24, 30, 60, 100])
def test_a_large_number_beside_others_does_not_hide_them(m, size):
    n, k, g = 1024, 1024, gen(size)
    a, w = torch.randn((m, k), generator=g, device=DEV), torch.randn((n, k), generator=g, device=DEV)
    a[:, 5::64] = 2.0 ** size
    w[:, 5::64] = 0.0
    assert ((ops.gemm_generic(a, w).double() - a.double() @ w.double().T).abs() <= bound(a, w)).all()


@pytest.mark.parametrize("m", [5, 70])
@pytest.mark.parametrize("sizes", [(-61, -61), (-100, 0), (-140, 100), (20, -140), (-40, -75), (60, 55), (110, 10), (61, 58)])
def test_small_and_large_operands(m, sizes):
    """Down to numbers without a leading one, up to sums near the largest float (those by multiply-adds, in 32 stretches of two
    chains); a result below 2^-126 is held to 2^-149."""
    n, k, g = 1024, 1024, gen(3)
    a = (torch.randn((m, k), generator=g, device=DEV).double() * 2.0 ** sizes[0]).float()
    w = (torch.randn((n, k), generator=g, device=DEV).double() * 2.0 ** sizes[1]).float()
    exact, got = a.double() @ w.double().T, ops.gemm_generic(a, w)
    terms = (a.double().abs() @ w.double().abs().T) * (16 + 32 + 3) * 2.0 ** -24
    assert ((got.double() - exact).abs() <= torch.maximum(bound(a, w), terms if sum(sizes) > 60 else 0 * terms) + 2.0 ** -149).all()


@pytest.mark.parametrize("m", [3, 32, 200])
def test_what_fits_into_32_bits_comes_out_exactly(m):
    k, g = 1024, gen(m)
    a = torch.randn((m, k), generator=g, device=DEV)
    assert torch.equal(ops.gemm_generic(a, torch.eye(k, device=DEV)), a)
    at, size = torch.randperm(k, generator=g, device=DEV), torch.exp2(torch.randint(-9, 9, (k, 1), generator=g, device=DEV).float())
    turned = torch.zeros((k, k), device=DEV)
    turned[torch.arange(k, device=DEV), at] = -size[:, 0]
    assert torch.equal(ops.gemm_generic(a, turned), -a[:, at] * size[:, 0])
    # one-hot rows of tokens
    hot = torch.zeros((m, k), device=DEV)
    hot[torch.arange(m, device=DEV), at[:m]] = 1.0
    w = torch.randn((1100, k), generator=g, device=DEV)
    assert torch.equal(ops.gemm_generic(hot, w), w[:, at[:m]].T)
    # whole numbers: of 8 bits, and of 12 and 10 bits with few that are not zero
    whole = lambda top, *shape: torch.randint(-top, top + 1, shape, generator=g, device=DEV).float()
    for x, y in ((whole(100, m, k), whole(100, 1100, k)), (whole(4000, m, k), whole(1000, 1100, k) * (torch.rand((1100, k), generator=g, device=DEV) < 0.002))):
        want = x.double() @ y.double().T
        assert want.abs().max() < 2 ** 24 and torch.equal(ops.gemm_generic(x, y).double(), want)


@pytest.mark.parametrize("k", [1024, 1500, 2048, 8192])
@pytest.mark.parametrize("kind", ["normal", "one sign", "wide", "few"])
def test_no_further_from_64_bits_than_multiply_adds(k, kind):
    n, g = 1100, gen(k)
    for m in (16, 200):
        a, w = torch.randn((m, k), generator=g, device=DEV), torch.randn((n, k), generator=g, device=DEV)
        if kind == "one sign":
            a, w = a.abs(), w.abs()
        elif kind == "wide":
            a = a * torch.exp2(torch.randn((m, k), generator=g, device=DEV) * 4)
        elif kind == "few":
            w = w * (torch.rand((n, k), generator=g, device=DEV) < 0.05)
        exact = a.double() @ w.double().T
        err = [float((got.double() - exact).norm() / exact.norm()) for got in (ops.gemm_generic(a, w), plain(a, w))]
        print(f"{kind}, {m} x {n} x {k}: {err[0]:.2e} on tensor cores, {err[1]:.2e} by multiply-adds")
        assert err[0] <= err[1]


def test_rows_that_are_no_numbers_leave_the_others_alone():
    """As a batch with sequences that have diverged: whole rows of NaN, of infinities and of what grows past the largest float."""
    m, n, k, g = 400, 2048, 2048, gen(8)
    a, w = torch.randn((m, k), generator=g, device=DEV), torch.randn((n, k), generator=g, device=DEV)
    a[10:140] = float("nan")
    a[150, 3], a[151, :] = float("nan"), float("inf")
    a[200:264, 77] = -float("inf")
    a[300] *= 2.0 ** 125
    got, want = ops.gemm_generic(a, w), plain(a, w)
    fine = torch.tensor([i for i in range(m) if not (10 <= i < 140 or i in (150, 151, 300) or 200 <= i < 264)], device=DEV)
    assert torch.isfinite(got[fine]).all() and torch.equal(got[fine], ops.gemm_generic(a[fine].contiguous(), w))
    odd = torch.tensor([i for i in range(m) if i not in set(fine.tolist())], device=DEV)
    assert torch.equal(torch.isnan(got[odd]), torch.isnan(want[odd])) and torch.equal(got[odd][want[odd].isinf()], want[odd][want[odd].isinf()])
    out = torch.ones((m, n), device=DEV)
    ops.gemm_generic(a, w, out=out, accumulate=True)
    assert torch.equal(out[fine], got[fine] + 1) and torch.equal(torch.isnan(out), torch.isnan(got))
    assert ops.gemm_f32_split_status() == 0


@pytest.mark.parametrize("m", [16, 256])
def test_tokens_that_hold_a_nan_cost_little(m):
    """A token with a NaN has no other results, and is read once by each warp that meets it: about twice the time of a product of finite
    numbers.  Working every result out by itself takes 30 times (few tokens) to 180 times as long."""
    n, k, g = 4096, 4096, gen(9)
    a, w = torch.randn((m, k), generator=g, device=DEV), torch.randn((n, k), generator=g, device=DEV)
    bad = a.clone()
    bad[:, 5] = float("nan")

    def best(x):
        times = []
        for _ in range(4):
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            start.record()
            got = ops.gemm_generic(x, w)
            end.record()
            torch.cuda.synchronize()
            times.append(start.elapsed_time(end))
        return min(times), got

    fine, _ = best(a)
    slow, got = best(bad)
    assert torch.isnan(got).all() and slow <= 6 * fine


@pytest.mark.parametrize("m", [1, 4, 65])
def test_the_kind_of_step_decides_between_the_kernels(m):
    n, k, g = 1100, 2048, gen(m)
    a, w = torch.randn((m, k), generator=g, device=DEV), torch.randn((n, k), generator=g, device=DEV)
    with ops.one_token_step(True):
        assert torch.equal(ops.gemm_generic(a, w), plain(a, w))
        with ops.one_token_step(False):
            assert not torch.equal(ops.gemm_generic(a, w), plain(a, w))
        assert torch.equal(ops.gemm_generic(a, w), plain(a, w))
    got = ops.gemm_generic(a, w)
    scratch = torch.empty((max(16, ops._bind().gi_gemm_f32_split_scratch(m, n, k)),), dtype=torch.uint8, device=DEV)
    split = torch.empty((m, n), device=DEV)
    assert ops._bind().gi_gemm_f32_split(split.data_ptr(), ops.GEMM_STORE, a.data_ptr(), w.data_ptr(), m, n, k, k, k, n, scratch.data_ptr(),
                                         scratch.numel(), ops._stream()) == 0
    assert torch.equal(got, split) and not torch.equal(got, plain(a, w))
    small = torch.randn((1023, k), generator=g, device=DEV)              # smaller matrices: multiply-adds in every step
    assert torch.equal(ops.gemm_generic(a, small), plain(a, small))


@pytest.mark.parametrize("m,launches", [(32, 1), (33, 2), (8192, 2), (8193, 4)])
def test_launches_are_counted(m, launches):
    a, w = torch.zeros((m, 1024), device=DEV), torch.zeros((1024, 1024), device=DEV)
    ops.gemm_generic(a, w)
    before = ops.launches
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        ops.gemm_generic(a, w)
        torch.cuda.synchronize()
    ours = [e for e in prof.events() if "split" in e.name and e.device_type == torch.autograd.DeviceType.CUDA]
    assert ops.launches - before == launches == len(ours)


@pytest.fixture(scope="module")
def wide_engine(tmp_path_factory):
    """Widths from which the prompts' products run on tensor cores."""
    from ghost_infer_b200.weights import write_random_model
    cfg = {"architectures": ["LlamaForCausalLM"], "hidden_size": 1024, "num_hidden_layers": 2, "num_attention_heads": 16,
           "num_key_value_heads": 8, "head_dim": 64, "intermediate_size": 1160, "vocab_size": 1300, "max_position_embeddings": 1024,
           "rope_theta": 10000.0, "rope_scaling": None, "rms_norm_eps": 1e-5, "tie_word_embeddings": False}
    d = str(tmp_path_factory.mktemp("wide_float32"))
    write_random_model(d, cfg, seed=6, dtype="float32", std=0.05, norm_jitter=0.1)
    return make_engine(d, "float32"), cfg


def rows_of(eng, steps):
    """Runs steps of (sequence, tokens) entries; the logits of every place of sequence 0."""
    slots, rows = {}, []
    for entries in steps:
        for i, _ in entries:
            if i not in slots:
                slots[i] = eng.cache.open_slot()
        out = eng.step([gi.StepEntry(slots[i], toks, list(range(len(toks))) if i == 0 else []) for i, toks in entries])
        if out is not None:
            rows.append(out.cpu().numpy())
    for s in slots.values():
        eng.cache.close_slot(s)
    return np.concatenate(rows)


def test_a_prompts_bits_do_not_depend_on_its_cut(wide_engine):
    eng, cfg = wide_engine
    me, mate = tokens_for(cfg, 150, 1), tokens_for(cfg, 400, 2)
    alone = rows_of(eng, [[(0, me)]])
    for size in (64, 33, 7, 2):
        assert np.array_equal(rows_of(eng, [[(0, me[i:i + size])] for i in range(0, 150, size)]), alone), f"pieces of {size}"
    assert np.array_equal(rows_of(eng, [[(1, mate), (0, me)]]), alone)
    # a piece of one token in a step that is a prompt step by its mate
    assert np.array_equal(rows_of(eng, [[(0, me[:100]), (1, mate[:300])], [(0, me[100:101]), (1, mate[300:310])], [(1, mate[310:]), (0, me[101:])]]), alone)


def test_a_one_token_steps_bits_do_not_depend_on_its_mates(wide_engine):
    eng, cfg = wide_engine
    me, mate = tokens_for(cfg, 60, 3), tokens_for(cfg, 60, 4)
    alone = rows_of(eng, [[(0, me[:40])]] + [[(0, [t])] for t in me[40:]])
    both = rows_of(eng, [[(0, me[:40]), (1, mate[:30])]] + [[(1, [u]), (0, [t])] for t, u in zip(me[40:], mate[30:])])
    assert np.array_equal(alone, both)
