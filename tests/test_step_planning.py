"""Host-side planning of a step: into how many slices of its context a decode step's attention cuts a sequence, which form a
prompt step over a latent cache takes."""
import random
from types import SimpleNamespace

import torch

from ghost_infer_b200.kernels import ops

BF, F32 = torch.bfloat16, torch.float32


def plan(n_seqs, max_kv_len, n_heads, n_kv, head_dim, window=None, dtype=BF, sms=148, kv_lens=None):
    return ops.attn_decode_plan(n_seqs, max_kv_len, sms, n_heads, n_kv, head_dim, window, dtype, kv_lens)


def test_slices_fill_the_blocks_an_sm_holds():
    # 8 sequences x 8 kv heads = 64 blocks per slice; two blocks per SM at head size 128, three at 64
    assert ops.attn_decode_blocks_per_sm(128, True) == 2 * ops.TUNE["attn_waves"]
    assert ops.attn_decode_blocks_per_sm(64, True) == 4 * ops.TUNE["attn_waves"]
    assert plan(8, 2048, 32, 8, 128) == (4, 0)
    assert plan(8, 4096, 32, 8, 64) == (9, 0)


def test_slices_are_never_shorter_than_256_positions_nor_more_than_32():
    assert plan(1, 100, 32, 8, 128) == (1, 0)
    assert plan(1, 300, 32, 8, 128) == (1, 0)
    assert plan(1, 600, 32, 8, 128) == (2, 0)
    assert plan(1, 1 << 20, 4, 1, 128) == (32, 0)
    # the length that counts is the longest sequence's now, not the end of its length bucket (which the plan must
    # still cover: it is kept until a sequence outgrows the bucket)
    assert plan(1, 4096, 32, 8, 128) == (16, 0)
    assert plan(1, 4096, 32, 8, 128, kv_lens=[2049]) == (8, 0)
    assert plan(2, 4096, 32, 8, 128, kv_lens=[300, 1100]) == (4, 0)


def test_many_equal_sequences_take_one_slice_each():
    # 64 sequences x 8 kv heads = 512 blocks for 296 places: cutting them would only add rounds
    assert plan(64, 2048, 32, 8, 128) == (1, 0)
    assert plan(64, 2048, 32, 8, 128, kv_lens=[2048] * 64) == (1, 0)
    # head size 64 with rings of two stages: four blocks per SM (the registers' limit), 592 places; equal lengths still
    # take one slice each
    assert ops.attn_decode_blocks_per_sm(64, True) == 4 * ops.TUNE["attn_waves"]
    assert plan(64, 1280, 32, 8, 64, kv_lens=[1200] * 64) == (1, 0)
    assert plan(18, 2048, 32, 8, 128) == (2, 0)                     # 144 blocks: two equal slices still fit one round


def test_many_unequal_sequences_can_be_cut_so_that_all_blocks_find_a_place_at_once(monkeypatch):
    """With TUNE["attn_own_slices"] and the lengths known: slices of a fixed number of tiles of each sequence's own span,
    the shortest (in steps of 256 keys) with which the blocks of all sequences fit the GPU at once.  The long sequences
    are cut, the short ones are not.  (Off by default: measured, the cut costs more than the evenness wins.)"""
    lens = [260 + 32 * i for i in range(64)]                        # 260 .. 2276
    assert plan(64, 4096, 32, 8, 64, kv_lens=lens) == (1, 0)
    monkeypatch.setitem(ops.TUNE, "attn_own_slices", True)
    n, own = plan(64, 4096, 32, 8, 64, kv_lens=lens)
    assert own > 0 and own % 16 == 0
    blocks = lambda o: sum(-(-(l + 64) // (o * 16)) for l in lens) * 8
    assert blocks(own) <= 592 < blocks(own - 16)                    # the shortest slice that fits
    assert n == -(-4096 // (own * 16))                              # the launch covers the longest a sequence may get
    assert max(lens) > own * 16                                     # the longest are cut
    # without the lengths nothing is known about them: one slice each
    assert plan(64, 4096, 32, 8, 64) == (1, 0)
    # more blocks than places even uncut: one slice each
    assert plan(64, 4096, 32, 8, 128, kv_lens=lens) == (1, 0)
    # padding rows of a recorded step count as a block each
    n2, own2 = plan(68, 4096, 32, 8, 64, kv_lens=lens)
    assert own2 >= own


def test_wide_groups_take_several_blocks_per_kv_head():
    # 40 heads on one kv head: three blocks of 16 rows per sequence and slice
    assert plan(4, 8192, 40, 1, 128) == ((2 * 148) // (4 * 3), 0)


def test_both_tensor_core_kernels_hold_the_same_number_of_blocks(monkeypatch):
    # keys on the rows, six warps with rings of two stages: 98 KB and up to 127 registers at head size 128, 50 KB and
    # 80 registers at 64; heads on the rows, four warps: the shared memory decides at 128, the registers at 64
    for on in (True, False):
        monkeypatch.setitem(ops.TUNE, "attn_keys_on_rows", on)
        assert ops.attn_decode_blocks_per_sm(128, True) == 2 * ops.TUNE["attn_waves"]
        assert ops.attn_decode_blocks_per_sm(64, True) == 4 * ops.TUNE["attn_waves"]


def test_head_sizes_the_tensor_core_kernel_declines_count_eight_rows_a_block():
    # head size 48 in bfloat16 runs the plain kernel: 8 heads a block (two blocks for a group of 16), two blocks per SM
    assert plan(4, 1 << 20, 32, 2, 48) == ((2 * 148) // (4 * 2 * 2), 0)
    assert plan(4, 1 << 20, 32, 2, 128) == (32, 0)


def test_32_bit_slices_follow_the_sequence_s_own_length():
    """In the 32-bit path a slice is eight 32-key tiles of the sequence's own span; the launch holds as many slices
    as the longest sequence needs, whatever the batch."""
    assert ops.OWN_LENGTH_TILES == 8
    assert plan(1, 256, 4, 2, 16, dtype=F32) == (1, 8)
    assert plan(1, 257, 4, 2, 16, dtype=F32) == (2, 8)
    assert plan(64, 257, 4, 2, 16, dtype=F32) == (2, 8)             # the batch does not matter
    assert plan(3, 5000, 4, 2, 16, dtype=F32) == ((5000 + 255) // 256, 8)
    # a window bounds the span: at most window + 31 keys from the tile the window starts in, plus that tile's head
    assert plan(3, 5000, 4, 2, 16, window=100, dtype=F32) == (1, 8)
    assert plan(3, 5000, 4, 2, 16, window=300, dtype=F32) == (2, 8)

# ---- prompt steps over a latent cache: which of the two forms, over how many rows ------------------------------------------
def prompt(pos0, lens, **kw):
    return SimpleNamespace(**{**dict(is_decode=False, n_seqs=len(lens), _host_pos0=list(pos0), _host_q_lens=list(lens), shared={}), **kw})


def test_rows_formed_per_head_are_those_the_kernels_count():
    """The gathering kernel and the attention lay a sequence's rows from the page of the first position that its first token
    sees to its last position; the buffers are as large as the host's count, which must be the same."""
    rng, chosen = random.Random(5), 0
    for _ in range(400):
        n = rng.randint(1, 5)
        pos0, lens = [rng.choice([0, rng.randint(1, 3000)]) for _ in range(n)], [rng.choice([1, rng.randint(1, 1500)]) for _ in range(n)]
        window = rng.choice([None, 1, 63, 64, 65, 500, rng.randint(1, 4000)])
        rows = tokens = pairs = tiles = 0
        for p, q in zip(pos0, lens):
            seen = [(max(0, i - window + 1) if window else 0, i) for i in range(p, p + q)]
            rows += p + q - seen[0][0] // 64 * 64
            pairs += sum(b - a + 1 for a, b in seen)
            tokens += q
            tiles = max(tiles, (max(b - a + 1 for a, b in seen) + 63) // 64)
        step = prompt(pos0, lens)
        assert ops._latent_visible(step, window) == (rows, pairs, tokens, tiles)
        got = ops.latent_expand_rows(step, 16, 128, 64, 128, 512, window, BF)
        assert got in (0, rows) and list(step.shared.values()) == [got]
        assert ops.latent_expand_rows(step, 16, 128, 64, 128, 512, window, BF) == got and len(step.shared) == 1
        chosen += got > 0
    assert 100 < chosen < 400


def test_what_keeps_a_prompt_on_the_latents():
    ask = lambda step, H=16, dim=128, rot=64, vdim=128, rank=512, window=None, dtype=BF: ops.latent_expand_rows(step, H, dim, rot, vdim, rank, window, dtype)
    step = prompt([0], [2048])
    assert ask(step) == 2048 and ask(step, dim=64, rot=16, vdim=8) == 2048
    for sizes in (dict(dim=96), dict(dim=32), dict(rot=0), dict(rot=24), dict(rot=80), dict(vdim=136), dict(vdim=20), dict(rank=508), dict(dtype=F32)):
        assert ask(step, **sizes) == 0
        assert not ops.latent_expand_sizes(**{**dict(dim=128, rot_dim=sizes.get("rot", 64), v_dim=sizes.get("vdim", 128), rank=512, dtype=BF), **{k: v for k, v in sizes.items() if k in ("dim", "rank", "dtype")}})
    assert ask(prompt([0], [2048], is_decode=True)) == 0
    assert ask(prompt([], [2048], n_seqs=1)) == 0 and ask(prompt([0], [2048], _host_pos0=None)) == 0
    assert ask(prompt([0], [8])) == 0                                  # a few tokens alone
    assert ask(prompt([3000], [16])) == 3016                           # and behind a long prefix
    rows = ops.LATENT_EXPAND_BYTES // (16 * 256 * 2)
    assert ask(prompt([rows - 500], [500])) == rows and ask(prompt([rows - 499], [500])) == 0
    assert ask(prompt([rows], [500]), window=1024) == rows + 500 - (rows - 1023) // 64 * 64
