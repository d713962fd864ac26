"""The C-ABI library without a GPU: it loads, exports every entry point that
include/axeng.h declares, keeps the reference's struct layout and op numbering,
and fails loudly (no CPU fallback) when no CUDA device is present."""
import ctypes
import os
import re

import numpy as np
import pytest

from axis_b200 import engine as E
from axis_b200._build import engine_lib

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib():
    return ctypes.CDLL(engine_lib())


def test_exports_match_header(lib):
    src = open(os.path.join(ROOT, "include", "axeng.h")).read()
    names = sorted(set(re.findall(r"\b(eng_[a-z0-9_]+)\s*\(", src)))
    assert len(names) >= 12
    for n in ("eng_init", "eng_alloc", "eng_has_flash", "eng_nccl_id", "eng_nccl_init", "eng_upload",
              "eng_download", "eng_run_plan", "eng_capture_plan", "eng_replay", "eng_sync", "eng_set_tf32"):
        assert n in names                      # the reference's twelve (axis/engine.py:81-100)
    for n in names:
        assert hasattr(lib, n), n


def test_struct_and_kind_numbering_match_reference():
    assert ctypes.sizeof(E._EngOp) == 80
    assert [f[0] for f in E._EngOp._fields_] == ["kind", "a", "b", "c", "d", "m", "n", "k", "batch", "tb",
                                                  "sa", "sb", "sc", "dt", "oa", "ob", "oc", "alpha", "beta", "gamma"]
    assert (E.GEMM, E.ADAMW, E.GEMM_SB, E.ROPE, E.CE, E.FLASH, E.FLASH_BWD, E.ALLREDUCE, E.BROADCAST) == \
        (0, 5, 8, 10, 20, 23, 25, 26, 31)
    src = open(os.path.join(ROOT, "include", "axeng.h")).read()
    for name, val in re.findall(r"ENG_([A-Z0-9_]+) = (\d+)", src):
        if name in E.KIND_NAMES:
            assert E.KIND_NAMES.index(name) == int(val), name
    o = E.op(E.GEMM_SB, a=1, b=2, c=3, m=4, n=5, k=6, tb=1, dt=2, alpha=0.5)
    pp = E.PackedPlan([o])
    raw = E._EngOp.from_buffer_copy(pp.arr.tobytes())
    assert (raw.kind, raw.a, raw.b, raw.c, raw.d, raw.m, raw.n, raw.k, raw.tb, raw.dt, raw.alpha) == \
        (8, 1, 2, 3, -1, 4, 5, 6, 1, 2, 0.5)


def test_bf16_conversion_is_round_to_nearest_even():
    a = np.array([1.0, 1.00390625, 1.01171875, -2.5, 3.3895314e38, 0.0], dtype=np.float32)
    b = E.bf16_bits_to_f32(E.f32_to_bf16_bits(a))
    assert b[0] == 1.0 and b[1] == 1.0 and b[2] == 1.015625 and b[3] == -2.5 and b[5] == 0.0


def _have_gpu():
    try:
        cu = ctypes.CDLL("libcuda.so.1")
        n = ctypes.c_int(0)
        return cu.cuInit(0) == 0 and cu.cuDeviceGetCount(ctypes.byref(n)) == 0 and n.value > 0
    except OSError:
        return False


@pytest.mark.skipif(_have_gpu(), reason="checks the no-device behaviour")
def test_no_device_means_loud_failure(lib):
    lib.eng_last_error.restype = ctypes.c_char_p
    assert lib.eng_init() != 0
    assert b"CUDA" in lib.eng_last_error()
    with pytest.raises(RuntimeError, match="engine init failed"):
        E.Engine()


def test_general_attention_allocates_what_its_cluster_merge_writes(lib):
    """A merge of attn_simt.cu lays out 4 rows x 32-column pieces x 256 threads of fp32 sums in a CTA's dynamic shared memory, and the
    forward a maximum and a sum for each of its 32 rows behind them, dK / dV two such arrays; the launch allocates no less."""
    f = lib.eng_attn_smem
    f.restype = ctypes.c_longlong
    for dh in range(1, 257):
        pieces = 1 if dh <= 32 else 2 if dh <= 64 else 4 if dh <= 128 else 8
        sums = 4 * pieces * 256 * 4
        for which, need in ((0, sums + 32 * 2 * 4), (1, sums), (2, 2 * sums)):
            assert need <= f(which, dh) <= 227 * 1024, (which, dh)
    assert f(0, 0) == f(2, 257) == f(3, 64) == -1


@pytest.mark.parametrize("B,H,T,DH,here", [
    # many short sequences: a 128-row tile is half empty and takes twice as long as the 64-row tiles of mma.sync
    (24, 16, 20, 64, 0), (24, 16, 64, 48, 0), (32, 30, 40, 64, 0), (24, 16, 65, 64, 1), (4, 24, 100, 64, 0), (18, 16, 128, 56, 0),
    # two tiles against three of mma.sync: not with a last wave that is less than half full
    (1, 1, 129, 64, 1), (4, 37, 129, 64, 1), (3, 50, 129, 64, 0), (7, 24, 192, 64, 0), (14, 16, 160, 64, 1), (8, 37, 129, 40, 1), (19, 32, 160, 64, 1),
    (3, 50, 193, 64, 1), (7, 24, 1000, 64, 1),
    (7, 24, 1000, 32, 0), (7, 24, 1000, 72, 0), (7, 24, 1000, 44, 0)])
def test_forward_attention_goes_where_it_is_faster(lib, B, H, T, DH, here):
    for kv in {1, H}:
        assert lib.eng_attn_route(0, B, H, kv, T, DH) == here


@pytest.mark.parametrize("B,H,KV,T,DH,here", [
    # one step for each key tile, or two for more key tiles than run at once
    (6, 32, 32, 20, 64, 0), (24, 16, 16, 64, 48, 0), (4, 24, 8, 64, 64, 0), (40, 8, 4, 3, 64, 1), (20, 16, 4, 64, 56, 1), (32, 30, 15, 40, 64, 0),
    (18, 16, 16, 65, 64, 1), (8, 37, 37, 65, 40, 1), (24, 16, 16, 129, 64, 0), (24, 16, 8, 129, 64, 1), (24, 16, 16, 193, 64, 1),
    # few steps: not with few 64-row tiles and short walks
    (1, 8, 4, 500, 64, 0), (1, 16, 8, 384, 56, 0), (1, 8, 8, 450, 64, 0), (1, 16, 2, 384, 56, 1), (1, 8, 8, 640, 56, 1), (4, 16, 16, 129, 64, 1),
    (4, 12, 4, 129, 64, 1), (1, 8, 4, 200, 64, 0), (1, 24, 8, 500, 64, 1), (3, 24, 8, 1000, 64, 1), (3, 24, 8, 1000, 72, 0), (3, 24, 8, 1000, 32, 0)])
def test_backward_attention_goes_where_it_is_faster(lib, B, H, KV, T, DH, here):
    assert (lib.eng_attn_route(1, B, H, KV, T, DH) > 0) == here


@pytest.mark.parametrize("B,H,KV,T,parts", [
    (2, 16, 2, 900, 4), (1, 12, 4, 2500, 2), (4, 24, 8, 500, 1), (2, 16, 2, 500, 4), (4, 12, 4, 129, 2), (1, 24, 8, 500, 4),
    # more clusters than run at once: a late one costs more than a shorter walk gains, unless the first tile's walk is the kernel
    (3, 12, 4, 384, 2), (1, 16, 8, 640, 2), (1, 8, 8, 1100, 2), (7, 24, 8, 129, 1), (1, 4, 2, 2500, 4), (1, 8, 4, 1100, 4), (2, 24, 8, 900, 2)])
def test_ctas_to_a_key_tile_of_the_attention_backward(lib, B, H, KV, T, parts):
    assert lib.eng_attn_route(1, B, H, KV, T, 64 if T % 128 else 56) == parts


@pytest.mark.parametrize("B,H,KV,T,parts64,parts128", [
    # short chains: the second CTA's set-up and the merge cost more than half a chain
    (22, 1, 1, 128, 1, 1), (4, 24, 12, 128, 1, 1), (2, 24, 12, 256, 1, 2), (13, 16, 4, 128, 1, 2), (1, 10, 10, 512, 2, 2), (2, 16, 4, 1024, 2, 4), (1, 16, 4, 1024, 4, 4),
    # one key tile to a head: no shorter walk for a cluster to wait for, beyond what runs at once not even for the longest chain
    (10, 16, 8, 128, 1, 1), (6, 64, 16, 128, 1, 1), (23, 12, 4, 128, 1, 1), (16, 128, 8, 128, 1, 1), (40, 32, 1, 128, 2, 2), (24, 32, 1, 128, 4, 4),
    # clusters that start late: only where the walks of the first round differ enough
    (16, 12, 4, 256, 1, 1), (12, 8, 4, 256, 1, 1), (22, 8, 2, 256, 1, 1), (13, 2, 2, 384, 1, 1), (6, 12, 4, 512, 1, 2), (25, 3, 1, 512, 1, 2), (11, 9, 3, 512, 1, 1), (3, 8, 8, 512, 1, 1),
    (7, 6, 3, 512, 1, 2), (20, 3, 1, 640, 2, 2), (2, 16, 8, 768, 2, 2), (6, 16, 4, 768, 2, 2), (7, 3, 1, 1536, 2, 2), (9, 2, 1, 2048, 2, 2), (2, 6, 2, 4096, 2, 2), (4, 24, 8, 768, 1, 1)])
def test_ctas_to_a_key_tile_of_whole_tiles(lib, B, H, KV, T, parts64, parts128):
    assert [lib.eng_attn_tile_parts(B, H, KV, T, dh) for dh in (64, 128)] == [parts64, parts128]
    assert lib.eng_attn_tile_parts(B, H, KV, T + 8, 64) == lib.eng_attn_tile_parts(B, H, KV, T, 96) == 0


@pytest.mark.parametrize("count,one_x,N,F,R,members,tokens,ctas", [
    # narrow inputs: a barrier and a sum across CTAs take as long as 500 columns
    (1, 1, 6510, 232, 8, 1, 32, 1), (1, 1, 9480, 160, 8, 1, 64, 1), (1, 0, 5241, 320, 16, 1, 32, 1), (3, 1, 615, 456, 8, 1, 32, 1), (2, 0, 4088, 288, 32, 1, 32, 1),
    (1, 0, 3196, 712, 16, 1, 32, 1), (1, 1, 45, 488, 8, 1, 32, 1), (3, 1, 302, 552, 16, 1, 32, 1),
    # members of a CTA: a long walk, or more products than a wave
    (3, 1, 2048, 4096, 16, 3, 64, 8), (2, 1, 3000, 2048, 16, 2, 64, 4), (3, 1, 4999, 776, 16, 1, 64, 1), (3, 1, 8572, 376, 8, 3, 64, 1), (3, 0, 8572, 376, 8, 1, 64, 1), (3, 1, 8192, 1536, 32, 3, 64, 2),
    # few blocks and long walks: 32 tokens, the columns over a cluster
    (1, 1, 70, 4096, 16, 1, 32, 8), (1, 1, 1024, 4096, 16, 1, 32, 8), (1, 1, 2048, 4096, 16, 1, 64, 8), (2, 1, 192, 1472, 32, 1, 32, 4), (1, 0, 4741, 1936, 16, 1, 64, 2), (1, 1, 8192, 4096, 16, 1, 64, 2)])
def test_cut_of_the_adapters_products(lib, count, one_x, N, F, R, members, tokens, ctas):
    cut = lib.eng_lora_proj_cut(count, one_x, N, F, R)
    assert (cut >> 16, cut >> 8 & 255, cut & 255) == (members, tokens, ctas)


@pytest.mark.parametrize("tb,m,n,k,batch,aligned,cut", [
    # few steps for 64-row tiles, or half of their rows empty, or steps that do not go evenly into the CTAs
    (0, 512, 256, 256, 1, 1, (64, 32, 8, 4)), (2, 512, 512, 256, 1, 1, (64, 32, 8, 2)), (1, 512, 256, 688, 1, 1, (64, 32, 8, 4)), (0, 512, 688, 256, 1, 1, (32, 32, 4, 1)),
    (0, 19, 1648, 176, 1, 1, (32, 32, 4, 1)), (1, 32, 1656, 144, 1, 1, (32, 32, 4, 1)), (0, 16, 2208, 320, 1, 1, (32, 32, 4, 2)), (2, 32, 528, 888, 1, 1, (32, 32, 4, 4)),
    (1, 704, 192, 176, 1, 1, (32, 32, 4, 1)), (1, 144, 2488, 184, 1, 1, (32, 32, 4, 1)), (0, 1104, 40, 384, 1, 1, (32, 32, 4, 2)), (0, 64, 984, 1168, 1, 1, (64, 32, 8, 8)),
    # shallow products of many tiles
    (0, 1184, 960, 24, 1, 1, (64, 64, 4, 1)), (1, 1968, 912, 16, 1, 1, (64, 64, 4, 1)), (0, 680, 2792, 32, 1, 1, (64, 64, 4, 1)), (1, 1552, 1176, 104, 1, 1, (64, 64, 4, 1)),
    (0, 1552, 1176, 104, 1, 1, (64, 64, 4, 1)), (0, 1264, 1108, 104, 1, 1, (64, 64, 8, 1)), (2, 1008, 656, 40, 1, 1, (32, 32, 4, 1)),
    # rows that are no whole 16-byte pieces
    (0, 1964, 456, 3179, 1, 1, (64, 64, 4, 1)), (1, 270, 2271, 220, 1, 1, (64, 64, 4, 1)), (2, 270, 2271, 220, 1, 1, (32, 32, 4, 1)), (0, 2422, 201, 324, 1, 1, (64, 32, 8, 1)), (0, 1547, 664, 34, 1, 1, (64, 64, 4, 1)), (0, 1453, 1051, 173, 1, 1, (64, 64, 4, 1)),
    (1, 1453, 1051, 173, 1, 1, (64, 64, 4, 1)), (1, 1613, 1101, 267, 1, 1, (64, 64, 8, 1)), (2, 1093, 1101, 267, 1, 1, (64, 64, 8, 1)), (2, 1146, 1651, 112, 1, 1, (64, 64, 4, 1)),
    # clusters that run at once; rounds of 64 x 64 tiles
    (1, 533, 228, 841, 1, 1, (32, 32, 4, 2)), (0, 560, 220, 612, 1, 1, (64, 32, 8, 4)), (1, 220, 258, 958, 1, 1, (32, 32, 4, 4)), (0, 128, 512, 1024, 1, 1, (64, 32, 8, 8)),
    (2, 2612, 864, 148, 1, 1, (64, 64, 4, 1)), (2, 2044, 1004, 764, 1, 1, (64, 64, 8, 1)), (0, 2732, 316, 88, 1, 1, (64, 64, 4, 1)), (1, 300, 1996, 84, 1, 1, (32, 32, 4, 1)), (2, 748, 1408, 96, 1, 1, (32, 32, 4, 1)), (2, 1744, 784, 92, 1, 1, (64, 64, 8, 1)), (0, 1115, 687, 51, 1, 1, (64, 64, 4, 1)), (1, 1032, 2085, 13, 1, 1, (128, 128, 8, 1)), (2, 2111, 2267, 12, 1, 1, (128, 128, 8, 1)),
    (1, 1679, 1771, 237, 1, 1, (128, 128, 8, 1)), (1, 1235, 2108, 701, 1, 1, (64, 64, 8, 1)), (0, 2111, 2267, 24, 1, 1, (64, 64, 4, 1)),
    (0, 215, 569, 2021, 1, 1, (32, 32, 4, 2)), (1, 202, 504, 677, 1, 1, (64, 32, 8, 4)), (0, 512, 256, 256, 1, 0, (32, 32, 4, 2)), (0, 1100, 1100, 100, 1, 1, (64, 64, 8, 1)),
    (0, 200, 200, 72, 19, 1, (64, 64, 8, 1)), (0, 1664, 1540, 96, 1, 1, (64, 64, 8, 1)), (0, 2000, 1700, 96, 1, 1, (128, 128, 8, 1)), (2, 2001, 1701, 40, 1, 1, (128, 128, 8, 1))])
def test_tiles_of_the_fp32_products(lib, tb, m, n, k, batch, aligned, cut):
    c = lib.eng_gemm_f32_cut(tb, m, n, k, batch, aligned)
    assert (c >> 20, c >> 8 & 0xfff, c >> 4 & 0xf, c & 0xf) == cut
    assert lib.eng_gemm_f32_cut(3, m, n, k, batch, aligned) == lib.eng_gemm_f32_cut(tb, 0, n, k, batch, aligned) == 0


def test_attention_route_of_invalid_shapes(lib):
    for a in ((0, 8, 4, 500, 64), (1, 0, 4, 500, 64), (1, 8, 0, 500, 64), (1, 8, 3, 500, 64), (1, 8, 4, 0, 64), (1, 8, 4, 500, 0)):
        assert lib.eng_attn_route(0, *a) == lib.eng_attn_route(1, *a) == 0


@pytest.mark.parametrize("B,H,KV,T,DH,parts", [
    (2, 8, 4, 256, 32, (4, 4, 8)), (1, 4, 1, 300, 64, (4, 4, 8)), (1, 2, 1, 225, 8, (4, 4, 8)), (16, 8, 8, 65, 64, (1, 1, 1)), (1, 8, 8, 16, 64, (1, 1, 1)),
    # one CTA of a wide head to an SM: none of two for each, unless a walk is long
    (3, 12, 12, 128, 256, (1, 1, 1)), (4, 8, 4, 100, 256, (1, 1, 2)), (1, 4, 1, 200, 256, (4, 4, 8)), (1, 16, 4, 400, 256, (2, 2, 8)), (8, 8, 2, 64, 256, (1, 1, 4)),
    # the third CTA of an SM is not worth a single tile
    (8, 16, 16, 64, 64, (1, 1, 1)), (32, 8, 4, 64, 32, (1, 1, 2))])
def test_ctas_to_a_walk_of_the_general_attention(lib, B, H, KV, T, DH, parts):
    assert tuple(lib.eng_attn_share(w, B, H, KV, T, DH) for w in range(3)) == parts


@pytest.mark.parametrize("B,H,KV,T,DH,ctas", [
    (2, 8, 4, 256, 32, (4, 4, 8)), (2, 16, 16, 333, 64, (4, 4, 4)), (40, 8, 2, 100, 48, (1, 1, 4)), (2, 8, 8, 130, 64, (4, 4, 4)),
    # one tile: nothing to share, and half of a block's rows empty
    (11, 1, 1, 13, 12, (1, 1, 0)), (3, 8, 8, 26, 12, (1, 1, 0)), (4, 1, 1, 27, 64, (1, 0, 0)), (240, 16, 4, 10, 48, (0, 0, 0)), (33, 12, 12, 17, 32, (0, 1, 1)), (1, 2, 1, 3, 64, (1, 0, 2)),
    # few blocks with long walks
    (1, 3, 1, 976, 16, (4, 0, 0)), (1, 8, 2, 928, 64, (4, 4, 0)), (6, 2, 1, 192, 12, (4, 4, 0)), (5, 1, 1, 73, 32, (4, 4, 4)),
    # not for these kernels
    (2, 8, 4, 256, 8, (0, 0, 0)), (2, 8, 4, 256, 34, (0, 0, 0)), (2, 8, 4, 256, 68, (0, 0, 0)), (2, 8, 3, 256, 64, (0, 0, 0)), (0, 8, 4, 256, 64, (0, 0, 0))])
def test_fp32_attention_goes_where_it_is_faster(lib, B, H, KV, T, DH, ctas):
    assert tuple(lib.eng_attn_f32_ctas(w, B, H, KV, T, DH) for w in range(3)) == ctas
    assert lib.eng_attn_f32_ctas(3, B, H, KV, T, DH) == 0


def test_cluster_barriers_are_met_by_converged_warps():
    """The aligned forms of the cluster barrier stand in one helper only, behind a __syncwarp(): lanes may come to them from a branch."""
    csrc = os.path.join(ROOT, "axis_b200", "csrc")
    found = []
    for f in sorted(os.listdir(csrc)):
        src = open(os.path.join(csrc, f)).read()
        found += [f] * src.count("barrier.cluster.arrive")
        if f == "common.cuh":
            assert re.search(r"void cluster_sync\(\) \{\s*__syncwarp\(\);\s*asm volatile\(\"barrier\.cluster\.arrive\.release\.aligned;", src)
    assert found == ["common.cuh"]
