"""The choices the Python face of the kernels makes before a launch: how many
blocks share the keys of a sequence, into how many slices of K a product is
cut, which product kernel takes which operands.  Pure arithmetic on shapes;
no GPU."""
import subprocess

import torch

from brolm_b200 import kernels
from brolm_b200.kernels import build


def test_decode_splits_make_one_wave_and_keep_two_pages_a_block():
    # Gemma 2 2B: 4 kv heads, 148 SMs
    assert kernels.decode_splits(8, 4, 8192, 0) == 4                 # 8 * 4 * 4 = 128 blocks
    assert kernels.decode_splits(1, 4, 8192, 0) == 37                # 148 blocks
    assert kernels.decode_splits(64, 4, 8192, 0) == 1                # more (sequence, head) pairs than SMs
    assert kernels.decode_splits(1, 4, 200, 0) == 2                  # four pages: two a block
    assert kernels.decode_splits(1, 4, 60, 0) == 1
    assert kernels.decode_splits(1, 1, 1 << 20, 0) == 40             # never more than the merge takes cheaply
    # a window bounds the keys a sequence has, whatever its length
    assert kernels.decode_splits(1, 4, 100000, 4096) == kernels.decode_splits(1, 4, 4096 + 63, 0)
    for batch in (1, 2, 3, 8, 20):
        for n_kv in (1, 4, 16):
            s = kernels.decode_splits(batch, n_kv, 8192, 0)
            assert 1 <= s <= 40 and (s == 1 or s * batch * n_kv <= 148)
    # sequences of very unequal lengths: several rounds of blocks, so that the SMs even them out
    assert kernels.decode_splits(16, 8, 8192, 0, sms=148, ragged=True) == 6       # 768 blocks, five rounds
    assert kernels.decode_splits(16, 8, 8192, 0, sms=148) == 1
    assert kernels.decode_splits(64, 4, 300, 0, sms=148, ragged=True) == 3        # two pages a block at least
    assert kernels.decode_splits(3, 4, 8192, 0, sms=148, ragged=True) == 40


def test_slices_of_k():
    x = torch.empty(8, 9216, dtype=torch.bfloat16)
    down = torch.empty(2304, 9216, dtype=torch.bfloat16)
    gate_up = torch.empty(18432, 2304, dtype=torch.bfloat16)
    assert kernels.skinny_parts(x, down, sms=148) == 3              # 144 blocks of 16 rows: three slices are one full round (432 of 444 places)
    assert kernels.skinny_parts(torch.empty(8, 2304, dtype=torch.bfloat16), gate_up) == 1
    # 27B down: 288 blocks, three slices are nearly two full rounds; two would leave a thin second round
    assert kernels.skinny_parts(torch.empty(8, 36864, dtype=torch.bfloat16), torch.empty(4608, 36864, dtype=torch.bfloat16), sms=148) == 3
    # 9B o: 224 blocks and a short K: one slice, a second round is not worth its start
    assert kernels.skinny_parts(torch.empty(16, 4096, dtype=torch.bfloat16), torch.empty(3584, 4096, dtype=torch.bfloat16), sms=148) == 1
    assert kernels.skinny_parts(torch.empty(8, 64, dtype=torch.bfloat16), torch.empty(16, 64, dtype=torch.bfloat16)) == 1
    # the fused q/k/v projection cannot be cut along K: 16-row tiles per block by how full the rounds get
    assert kernels.skinny_rope_tiles(4096, 2304, sms=148) == 1       # 2B: 256 blocks, three to an SM
    assert kernels.skinny_rope_tiles(8192, 3584, sms=148) == 2       # 9B: 512 would be a round and a thin one; 256 of two tiles
    assert kernels.skinny_rope_tiles(48, 64, sms=148) == 1           # an odd number of tiles
    p = kernels.gemm_stream_parts(x, down)
    assert p >= 1 and p * 18 >= 100                                  # 18 row tiles: enough (tile, slice) items for the SMs


def test_which_product_takes_which_operands():
    w = torch.empty(4096, 2304, dtype=torch.bfloat16)
    few, many = torch.empty(8, 2304, dtype=torch.bfloat16), torch.empty(2048, 2304, dtype=torch.bfloat16)
    assert kernels.skinny_ok(few, w) and not kernels.skinny_ok(many, w)
    assert kernels.skinny_ok(torch.empty(16, 2304, dtype=torch.bfloat16), w)
    assert not kernels.skinny_ok(torch.empty(17, 2304, dtype=torch.bfloat16), w)
    assert not kernels.skinny_ok(few.float(), w)                      # bfloat16 only
    # the tcgen05 product wants a tile for every SM
    assert kernels.gemm_tc_ok(many, w)                                # 16 x 16 = 256 tiles
    assert not kernels.gemm_tc_ok(many, torch.empty(2304, 2304, dtype=torch.bfloat16))      # 16 x 9 = 144
    assert not kernels.gemm_tc_ok(few, w)
    assert not kernels.gemm_tc_ok(torch.empty(2048, 2308, dtype=torch.bfloat16)[:, :2301], w[:, :2301])   # K % 8
    # the weight stream takes up to 128 rows
    assert kernels.gemm_stream_ok(torch.empty(128, 2304, dtype=torch.bfloat16), w)
    assert not kernels.gemm_stream_ok(torch.empty(129, 2304, dtype=torch.bfloat16), w)
    # the tcgen05 prompt attention: head sizes 64, 128, 256 and groups that divide 128
    assert kernels.attention_prefill_tc_ok(256, 2) and kernels.attention_prefill_tc_ok(128, 8)
    assert not kernels.attention_prefill_tc_ok(80, 2) and not kernels.attention_prefill_tc_ok(128, 3)


def test_float_attention_shares_as_many_spans_as_a_tile_can_see():
    """Pages bound the keys only where positions never go round; a window or a chunk bounds them otherwise, wherever it
    lies over the spans."""
    assert kernels.attn_f32_max_keys(448, 1 << 30) == 448 and kernels.attn_f32_max_keys(192, 256) == 192
    assert kernels.attn_f32_max_keys(256, 256) is None and kernels.attn_f32_max_keys(512, 256) is None
    for window in (1, 65, 128, 129, 200, 256, 300):
        ring = -(-window // 64) * 64
        for group in (1, 4, 8, 40):
            splits = kernels.attn_f32_splits(1, 1, group, 64, 1, 1, kernels.attn_f32_max_keys(ring, ring), window)
            for pos in range(1000):
                seen = pos // kernels.F32_SPAN - max(0, pos - window + 1) // kernels.F32_SPAN + 1
                assert splits == 0 or seen <= splits, (window, group, pos)


def test_decode_splits_where_two_blocks_share_an_sm():
    two = dict(sms=148, per_sm=kernels.decode_blocks_per_sm(256))
    assert kernels.decode_blocks_per_sm(128) == 1 and two["per_sm"] == 2
    assert kernels.decode_splits(8, 4, 8192, 0, **two) == 9                       # 288 blocks for 296 places
    assert kernels.decode_splits(1, 4, 8192, 0, **two) == 37                      # 40 would be little more than one round
    assert kernels.decode_splits(64, 4, 2048, 0, **two) == 1
    assert kernels.decode_splits(8, 4, 2048, 0, **two) == 4                       # nine would be runs of three or four pages
    assert kernels.decode_splits(8, 4, 4096, 0, **two) == 9
    assert kernels.decode_splits(12, 4, 8192, 0, **two) == 3                      # 144 blocks keep all SMs busy
    assert kernels.decode_splits(16, 8, 1024, 0, **two) == 1 and kernels.decode_splits(16, 8, 2048, 0, **two) == 2
    assert kernels.decode_splits(12, 8, 1024, 0, **two) == 3                      # 96 of 148 SMs busy
    assert kernels.decode_splits(36, 4, 8192, 0, **two) == 2 and kernels.decode_splits(36, 4, 2048, 0, **two) == 1
    assert kernels.decode_splits(16, 8, 8192, 0, ragged=True, **two) == 5
    assert kernels.decode_splits(3, 4, 700, 0, **two) == kernels.decode_splits(3, 4, 700, 0, sms=148)
    for batch in (1, 2, 3, 5, 8, 13, 16, 30, 64):
        for keys in (60, 300, 1280, 8192):
            assert 1 <= kernels.decode_splits(batch, 4, keys, 0, **two) <= max(1, ((keys + 63) // 64 + 1) // 2)


def test_which_few_token_products_stream(monkeypatch):
    monkeypatch.setattr(kernels, "gemm_stream_ok", lambda x, w: True)             # (tensors without memory have no address)
    like = lambda *shape: torch.empty(shape, dtype=torch.bfloat16, device="meta")
    of = lambda M, N, K: kernels.stream_instead_of_skinny(like(M, K), like(N, K), sms=148)
    assert of(1, 28672, 3584) and of(16, 73728, 4608)                 # 9B, 27B gate and up
    assert not of(16, 18432, 2304) and not of(8, 8192, 2048)          # no more pieces than SMs
    assert of(8, 73728, 4608) and not of(1, 73728, 4608) and not of(7, 57344, 4096)     # several rounds: not for the fewest
    assert not of(8, 128 * 300, 512)                                        # a second round of four pieces
    slices = lambda N, K: kernels.gemm_stream_parts(like(16, K), like(N, K), sms=148)
    assert slices(3584, 14336) == 10 and slices(8192, 3584) == 4 and slices(2304, 9216) == 8


def test_partial_sums_of_the_float_product_are_bounded():
    """A cut along K pays for the sums it writes and reads again, and never takes more than a fixed scratch."""
    assert kernels.linear_f32_slices(9216, 18) == 1 and kernels.linear_f32_slices(9216, 1) == 18
    assert kernels.linear_f32_slices(9216 + 4, 9) == 11
    cuts = 0
    for M in (17, 40, 300, 1024, 4096, 4196, 8192, 16384):
        for N, K in ((2304, 2304), (2304, 9216), (3584, 14336), (4608, 36864), (36864, 4608), (256000, 2304), (64, 100)):
            cut = kernels.linear_f32_plan(M, N, K, 148)[1]
            assert 0 <= cut < -(-K // kernels.F32_SEGMENT)
            if cut:
                cuts += 1
                assert kernels.linear_f32_slices(K, cut) * M * N * 4 <= 256 << 20, (M, N, K, cut)
    assert cuts > 10


def test_slices_of_the_float_product_on_tensor_cores():
    """None is empty, each is whole stages of 64, clusters of at most eight; small weights are not for it."""
    for N in (64, 1100, 4100, 18432, 256000):
        for K in list(range(248, 3000, 4)) + [9216, 14336, 36864]:
            n = kernels.linear_f32_tc_slices(N, K)
            assert n in (0, 1, 2, 4, 8) and (n > 0) == (N * K >= 1 << 20 and K >= 256)
            if n:
                per = kernels._f32_tc_slice(K, n)
                assert per % 64 == 0 and (n - 1) * per < K <= n * per and (n == 1 or -(-N // 128) * n <= 148)


def test_where_the_slices_of_a_float_product_are_added():
    """By a kernel behind it where clusters of eight blocks would queue for room, as long as the sums take no more than 256 MB."""
    scratch = kernels.linear_f32_tc_scratch
    assert scratch(3, 2304, 8) and scratch(32, 2176, 8) and not scratch(3, 2048, 8) and not scratch(3, 4096, 4)
    assert scratch(33, 1024, 8) and scratch(300, 2304, 8) and not scratch(3000, 2304, 8)
    assert scratch(32, 2304, 8) and not scratch(10400, 128, 8) and not scratch(9000, 1024, 8)


def test_which_kernel_takes_a_float_product():
    """Streams for few rows, small tiles where large ones leave SMs idle, large ones where there are enough of them."""
    plan = lambda M, N, K: kernels.linear_f32_plan(M, N, K, 148)
    assert plan(1, 2304, 9216) == plan(16, 2304, 2304) == plan(1, 16, 16) == (1, 0)
    assert plan(12, 100, 100) == (32, 0)                         # too short a K for streams
    assert plan(8, 16, 16) == plan(300, 16, 16) == plan(64 * 65535, 16, 16) == (0, 0)
    assert plan(64 * 65535 + 1, 16, 16)[0] in (32, 64)           # more rows than that kernel's grid holds
    assert plan(300, 64, 64) == plan(100, 2304, 256) == (32, 0)
    assert plan(100, 256, 1024) == (32, 1)
    assert plan(2048, 2304, 9216) == plan(300, 18432, 2304) == (64, 0)
    assert plan(300, 2304, 9216) == (64, 1)


def test_what_belongs_to_a_device_is_done_for_each(tmp_path):
    """A limit raised on one device says nothing of another, and a call that failed is made again."""
    (tmp_path / "t.cpp").write_text("""
#include "once_per_device.h"
#include <cstdio>
#include <initializer_list>
int main() {
    OncePerDevice once;
    int calls[70] = {}, failing = 1;
    auto on = [&](int d) { return once.run(d, [&] { ++calls[d + 1]; return d == 3 ? failing : 0; }); };
    int bad = 0;
    for (int round = 0; round < 3; ++round)
        for (int d : {0, 1, 63, 64, -1}) bad += on(d) != 0;
    bad += on(3) != 1; failing = 0; bad += on(3) != 0; bad += on(3) != 0;
    std::printf("%d %d %d %d %d %d", bad, calls[1], calls[2], calls[64], calls[65], calls[4]);
}
""")
    subprocess.run(["g++", "-std=c++17", "-I", build.CSRC, "-o", str(tmp_path / "t"), str(tmp_path / "t.cpp")], check=True)
    assert subprocess.run([str(tmp_path / "t")], capture_output=True, text=True, check=True).stdout == "0 1 1 1 3 2"


def test_decode_blocks_start_by_length_only_where_runs_are_long():
    first = kernels.decode_longest_first
    assert not first(False, 1, 8192, 0, 256)                                      # equal lengths keep their own order
    assert first(True, 5, 8192, 0, 256) and first(True, 2, 1024, 0, 256)
    assert not first(True, 6, 1024, 0, 256) and not first(True, 1, 256, 0, 256)
    assert not first(True, 1, 8192, 64, 256) and first(True, 1, 8192, 4096, 256)  # a window bounds a run, too
    assert not first(True, 2, 1024, 0, 128) and first(True, 2, 4096, 0, 128)


def test_streams_are_nobody_elses_until_given_back(monkeypatch):
    made = []
    monkeypatch.setattr(kernels, "_free_streams", {})
    monkeypatch.setattr(kernels, "_new_stream", lambda index: made.append(index) or object())
    a, b, c = kernels.take_stream(0), kernels.take_stream(0), kernels.take_stream(1)
    assert len({id(a), id(b), id(c)}) == 3 and made == [0, 0, 1]
    kernels.give_stream(0, a)
    assert kernels.take_stream(1) is not a and kernels.take_stream(0) is a
    assert len(made) == 4


def test_float_attention_shares_spans_only_where_the_merge_is_worth_it():
    worth = lambda *a, **kw: kernels.attn_f32_worth_sharing(*a, sms=148, **kw)
    assert worth(1, 4, 2, 256, 256, 300, 300) and worth(3, 4, 2, 256, 256, 1, 512) and worth(64, 4, 2, 256, 256, 1, 512)
    assert not worth(1, 4, 2, 256, 256, 100, 100) and not worth(1, 4, 2, 256, 256, 1, 128)     # one span
    assert not worth(1, 2, 2, 32, 32, 300, 300, window=16) and not worth(1, 8, 4, 128, 128, 300, 300, window=64)
    assert worth(1, 4, 2, 256, 256, 300, 300, window=100) and not worth(32, 8, 4, 128, 128, 1, 256)
    assert not worth(1, 4, 2, 256, 256, 1, None)                                               # no bound
    # up to one span an SM in clusters: worth it for the smallest heads, too; beyond, what a block a span takes decides
    assert worth(8, 2, 2, 16, 16, 1, 200) and worth(32, 1, 8, 64, 64, 1, 200) and worth(3, 4, 2, 256, 256, 1, 200)
    assert not worth(128, 2, 2, 16, 16, 1, 200) and not worth(8, 2, 2, 16, 16, 1, 120)


def test_float_attention_is_cut_by_the_lengths_not_by_the_table():
    """A page table for 32,768 tokens and sequences of at most 512: four spans, not 256, and no more scratch than for those."""
    bound = kernels.attn_f32_max_keys
    assert bound(32768, 1 << 30, 512) == 512 and bound(32768, 1 << 30) == 32768 and bound(256, 1 << 30, 512) == 256
    assert bound(256, 256, 300) == 300 and bound(256, 256) is None and bound(256, 256, 0) is None
    splits = lambda keys, batch: kernels.attn_f32_splits(batch, 4, 2, 256, batch, 1, keys, sms=148)
    assert splits(bound(32768, 1 << 30, 512), 3) == 4
    assert splits(bound(32768, 1 << 30, 512), 32) == 4 and splits(bound(32768, 1 << 30), 32) == 0
