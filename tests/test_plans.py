"""Launch plans over ranges of sizes. Host code: no GPU is needed."""
import ctypes

import pytest

SMS = 148


def _int4_plan(M, N, K, split_k, sms=SMS):
    from flydsl_b200 import _lib

    plan = (ctypes.c_int32 * 5)()
    _lib.check(_lib.load().flyb200_int4_plan(M, N, K, split_k, sms, plan))
    return tuple(plan)


@pytest.mark.parametrize("M", [1, 16, 17, 32, 33, 64])
@pytest.mark.parametrize("split_k", [0, 1, 3, 8])
def test_int4_ring_slots_belong_to_one_set(M, split_k):
    """A consumer warp waits for the fills of the groups that its set takes. Parity waits are sound only
    if it sees every fill of a slot, so no slot may hold groups of two sets."""
    wrapped = 0
    for N in range(128, 16385, 384):
        for K in range(128, 16385, 128):
            _, sets, splits, groups, slots = _int4_plan(M, N, K, split_k)
            if splits == 0:   # no plan: the call is refused
                continue
            assert sets in ((1, 2) if M <= 32 else (1,)) and 2 <= slots <= 16
            owner = {}
            for g in range(groups):
                assert owner.setdefault(g % slots, g % sets) == g % sets, (N, K, sets, groups, slots)
            wrapped += groups > slots
    assert wrapped > 100


@pytest.mark.parametrize("M", [1, 16, 17, 32, 33, 64])
def test_int4_two_sets_only_where_every_cta_has_an_sm(M):
    """A CTA with two sets of warps fills an SM: no second wave, and enough groups for both sets."""
    seen = set()
    for N in range(128, 24577, 128):
        for K in range(128, 16385, 256):
            mb, sets, splits, groups, slots = _int4_plan(M, N, K, 0)
            ctas = N // 128 * splits
            seen.add(sets)
            if sets == 2:
                assert ctas <= SMS and groups >= 6
            else:   # two CTAs of up to 32 tokens share an SM's shared memory
                slot, rest = 8192 + mb * 4096, (16 * mb + 8) * 512 + groups * 256 + 2048
                assert slots * slot + rest + 1024 <= 233472 // (2 if M <= 32 else 1)
    assert seen == ({1, 2} if M <= 32 else {1})


def _int4_tensor_plan(M, N, K, split_k=0, sms=SMS):
    from flydsl_b200 import _lib

    plan = (ctypes.c_int32 * 7)()
    _lib.check(_lib.load().flyb200_int4_tensor_plan(M, N, K, split_k, sms, plan))
    return dict(zip(("kernel", "cols", "splits", "groups", "slots", "smem", "tmem"), plan))


@pytest.mark.parametrize("M", [1, 16, 17, 32, 33, 64])
@pytest.mark.parametrize("split_k", [0, 1, 3, 8])
def test_int4_tensor_rings(M, split_k):
    """The tcgen05 kernel's plans. A ring that wraps is even, so that a slot's groups all belong to one of the two sets
    of dequantisers (see test_int4_ring_slots_belong_to_one_set); it fits the SM, or half of it where two CTAs are to
    share one; the groups of a cluster cover K; and every size has a plan for one of the two kernels."""
    wrapped, kernels = 0, set()
    for N in range(128, 16385, 768):
        for K in list(range(128, 16385, 128)) + list(range(16512, 131072, 3200)):
            plan = _int4_tensor_plan(M, N, K, split_k)
            if plan["splits"] == 0:
                assert plan["kernel"] == 1
            else:
                groups, slots = plan["groups"], plan["slots"]
                assert plan["cols"] == (16 if M <= 16 else 32 if M <= 32 else 64)
                assert min(2, groups) <= slots <= min(16, groups) and (slots == groups or slots % 2 == 0)
                assert (plan["splits"] - 1) * groups < K // 128 <= plan["splits"] * groups
                assert plan["smem"] <= 232448
                if M <= 32 and groups <= 64:
                    assert 2 * (plan["smem"] + 1024) <= 233472
                wrapped += groups > slots
                assert M <= 32 or plan["kernel"] == 2
            if plan["kernel"] == 1 and split_k == 0:
                assert _int4_plan(M, N, K, 0)[2] > 0
            kernels.add(plan["kernel"])
    assert wrapped > 100 and 2 in kernels and (M > 32 or 1 in kernels)


def _decode_plan(M, N, K, split_k=0, sms=SMS):
    from flydsl_b200 import _lib

    plan = (ctypes.c_int32 * 6)()
    _lib.check(_lib.load().flyb200_decode_plan(M, N, K, split_k, sms, plan))
    return dict(zip(("cols", "splits", "groups", "stages", "smem", "tmem"), plan))


@pytest.mark.parametrize("plan_of", [_int4_tensor_plan, _decode_plan])
@pytest.mark.parametrize("split_k", [0, 1, 8])
def test_resident_ctas_of_cluster_kernels_find_their_tensor_memory(plan_of, split_k):
    """A CTA takes its columns of tensor memory by an instruction that waits without a limit, and then meets its cluster.
    Two streams could wait for one another's columns in a circle unless shared memory (228 KB an SM, 1 KB of it taken by
    every CTA) keeps CTAs apart that ask for more than the 512 columns together: registers do so by chance only."""
    seen = set()
    for M in (1, 16, 17, 32, 33, 64):
        for N in (128, 1024, 8192, 24576):
            for K in (128, 256, 512, 1024, 2048, 4096, 8192, 32768):
                plan = plan_of(M, N, K, split_k)
                if plan["splits"]:
                    assert (plan["smem"] + 1024) * 512 >= 233472 * plan["tmem"], (M, N, K, plan)
                    assert plan["smem"] <= 232448
                    seen.add(plan["tmem"])
    assert seen == ({64, 128, 256} if plan_of is _decode_plan else {256, 512})


# M, N, K; time (us) of the mma.sync kernel, of the tcgen05 one (graph replays, cold weights)
INT4_SIZES = [
    (11, 20480, 256, 4.2, 4.8), (14, 4096, 3328, 6.9, 5.5), (13, 7552, 2048, 6.7, 5.7), (2, 2688, 4608, 6.1, 5.2),
    (8, 6656, 1280, 4.7, 5.4), (13, 6656, 1152, 5.0, 5.5), (32, 17664, 384, 5.4, 5.9),
    (3, 30080, 512, 7.4, 5.9), (5, 2048, 5632, 7.2, 5.9), (4, 768, 8320, 6.7, 5.7), (1, 128, 9216, 6.1, 5.1),
    (15, 6144, 1664, 7.0, 5.9), (20, 768, 3712, 5.6, 4.6), (20, 16000, 128, 3.6, 4.7), (18, 10880, 256, 4.2, 4.8),
    (22, 2048, 4352, 7.9, 5.5), (29, 16640, 256, 4.9, 5.5), (28, 5504, 1792, 6.5, 6.0), (55, 256, 768, 5.9, 5.4),
    (34, 4096, 512, 5.5, 4.9), (58, 1024, 4608, 9.7, 6.4)
]


@pytest.mark.parametrize("M,N,K,stream_us,tensor_us", INT4_SIZES)
def test_int4_takes_the_kernel_that_measured_faster(M, N, K, stream_us, tensor_us):
    assert _int4_tensor_plan(M, N, K)["kernel"] == (1 if stream_us < tensor_us else 2)


def _kernel_source(name):
    import os
    import re

    from flydsl_b200 import build

    text = open(os.path.join(build.CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", text)


@pytest.mark.parametrize("name", ["blockscale_gemm.cu", "moe_swap.cu", "pt_pair_gemm.cu", "bs_pair_gemm.cu"])
def test_roles_that_may_give_up_meet_at_bounded_barriers_only(name):
    """In these kernels a warp whose bounded wait runs out leaves its loop at once, so nobody may wait for
    it at a named hardware barrier, which has no limit (decode_gemm.cu, int4_gemm.cu and int4_stream.cu send
    the warps that gave up through theirs). __syncthreads is reached by every warp on every path."""
    import re

    source = _kernel_source(name)
    assert "mbar_wait" in source
    assert not re.search(r"\bbar(rier)?\.(cta\.)?sync", source)


def test_split_k_cta_that_gave_up_outlives_the_copies_sent_to_it():
    """A sender leaves once every CTA of its cluster has arrived at the last cluster barrier, and its copies
    read its shared memory until they land. So an owner that no longer waits for them (it gave up) has to
    pause before that barrier: behind it the sender may be gone."""
    source = _kernel_source("blockscale_gemm.cu")
    end = source[source.index("if (warp < kEpiWarp0) cluster_sync_all();"):]
    end = end[:end.index("__syncthreads();")]
    assert end.index("drain_if_aborted();") < end.rindex("cluster_sync_all();")


def _gemm_plan(M, N, K, pertoken=False, sms=SMS, **cfg):
    from flydsl_b200 import _lib

    cfg = _lib.GemmCfg(*[cfg.get(name, 0) for name in ("block_n", "max_ctas", "path", "split_k")])
    plan = (ctypes.c_int32 * 5)()
    _lib.check(_lib.load().flyb200_gemm_plan(int(pertoken), M, N, K, ctypes.byref(cfg), sms, plan))
    return dict(zip(("kernel", "block_n", "splits", "kbps", "ctas"), plan))


TILED, DECODE, PAIR = 1, 2, 3


def test_requests_of_the_caller_are_honoured():
    wide = dict(M=16, N=16384, K=2048)
    assert _gemm_plan(**wide)["kernel"] == TILED
    # a cluster size or a limit on the CTAs was asked for: the route of these calls is the decode kernel
    assert _gemm_plan(**wide, split_k=1)["kernel"] == DECODE
    assert _gemm_plan(**wide, max_ctas=64)["kernel"] == DECODE
    # the limit on the CTAs holds with a split as well
    for pertoken in (False, True):
        deep = dict(M=256, N=1024, K=8192, pertoken=pertoken, path=TILED, split_k=4)
        free = _gemm_plan(**deep)
        assert free["splits"] == 4 and free["ctas"] > 8
        for limit in (1, 5, 8, free["ctas"] - 1, free["ctas"], 148, 1000):
            plan = _gemm_plan(**deep, max_ctas=limit)
            assert plan["ctas"] <= limit and (plan["splits"] == 4) == (limit >= free["ctas"])
        assert _gemm_plan(256, 1024, 8192, pertoken, max_ctas=8)["ctas"] <= 8
        # path 0 with some request made stays unsplit, as the tiled kernel always was then
        assert _gemm_plan(256, 1024, 8192, pertoken)["splits"] > 1
        assert _gemm_plan(256, 1024, 8192, pertoken, split_k=4)["splits"] == 1


def test_plan_refuses_what_the_call_refuses():
    bad = [dict(M=0, N=128, K=128), dict(M=1, N=8, K=128), dict(M=1, N=24, K=128), dict(M=1, N=128, K=192),
           dict(M=65, N=128, K=128, path=DECODE), dict(M=1, N=128, K=128, path=4),
           dict(M=1, N=128, K=128, path=PAIR), dict(M=255, N=256, K=128, path=PAIR, pertoken=True)]
    for case in bad:
        with pytest.raises(ValueError):
            _gemm_plan(**case)


def _moe_layer(E, H, I, topk, tile_m, mode="reduce"):
    import torch

    from flydsl_b200.moe import BlockscaleMoE

    def meta(*shape, dtype=torch.float8_e4m3fn):
        return torch.empty(shape, dtype=dtype, device="meta")

    return BlockscaleMoE(meta(E, 2 * I, H), meta(E, 2 * I // 128 * (H // 128), dtype=torch.float32), meta(E, H, I),
                         meta(E, H // 128 * (I // 128), dtype=torch.float32), topk=topk, tile_m=tile_m, mode=mode)


@pytest.mark.parametrize("E,H,I,topk,tile_m,least", [
    (256, 7168, 2048, 8, 16, 12), (256, 7168, 2048, 8, 32, 12),           # from 4 GB of weights in use on
    (128, 4096, 1536, 8, 16, 26), (128, 4096, 1536, 8, 32, 256),          # routes for 0.1 / 0.5 of all blocks
    (64, 2048, 1024, 6, 16, 128), (64, 2048, 1024, 6, 32, 256), (128, 2048, 512, 2, 8, 384)])   # small layers: 0.75
def test_moe_small_blocks_take_routing_order_where_it_pays_off(E, H, I, topk, tile_m, least):
    layer = _moe_layer(E, H, I, topk, tile_m)
    for T in range(1, 1025):
        assert layer._small_pays_off(T) == (T >= least), T


def test_moe_more_blocks_than_the_kernel_lists():
    wide, narrow = _moe_layer(128, 1024, 256, 8, 32), _moe_layer(128, 1024, 256, 8, 16)
    assert wide._small_pays_off(15873) and not wide._small_pays_off(15874)   # 4096 blocks, one more
    assert narrow._small_pays_off(100000)


# stage, routing order, blocks, output channels; time (us) in 128- and in 256-wide tiles
MOE_WIDTHS = [
    (1, 0, 50, 384, 24.5, 19.4), (1, 0, 67, 384, 23.5, 19.9), (1, 0, 38, 512, 11.9, 9.9), (1, 1, 69, 384, 26.8, 31.6),
    (1, 1, 37, 768, 44.0, 50.5), (1, 1, 33, 1920, 30.9, 26.9), (2, 0, 68, 3840, 34.5, 24.1), (2, 0, 25, 2176, 8.6, 6.8),
    (2, 0, 38, 1024, 9.1, 7.1), (2, 1, 9, 4736, 14.3, 19.0), (2, 1, 34, 5760, 33.0, 26.8), (2, 1, 72, 1536, 17.1, 13.0)
]


@pytest.mark.parametrize("stage,a_sorted,blocks,n,us_128,us_256", MOE_WIDTHS)
def test_moe_stage_takes_the_width_that_measured_faster(stage, a_sorted, blocks, n, us_128, us_256):
    from flydsl_b200 import _lib

    width = ctypes.c_int32(0)
    _lib.check(_lib.load().flyb200_moe_plan(stage, n, blocks, a_sorted, SMS, width))
    assert width.value == (128 if us_128 < us_256 else 256)


@pytest.mark.parametrize("mode", ["reduce", "atomic"])
@pytest.mark.parametrize("tile_m", [8, 16, 32])
def test_moe_layer_scratch_is_bounded_over_token_counts(tile_m, mode):
    """A server's decode batches, every size from 1 to 512, on a layer of the benchmark's size."""
    import torch

    from flydsl_b200 import moe

    E, H, I, topk, dev = 256, 7168, 2048, 8, torch.device("meta")
    layer = _moe_layer(E, H, I, topk, tile_m, mode)
    for T in range(1, 513):
        b = layer._buffers(T, dev, True)
        rows = T * topk + E * tile_m - topk
        assert b["rows"] == rows and b["x_sorted"].shape == (rows, H) and b["out1"].shape == (rows, I)
    kept = sum(t.numel() * t.element_size() for b in layer._buf.values() for t in b.values() if torch.is_tensor(t))
    assert 0 < kept <= moe._KEPT_SMALL_BYTES
    first = layer._buffers(1, dev, True)
    assert layer._buffers(1, dev, True) is first   # the sizes met first keep theirs


# M, N, K; time (us) on the decode kernel, on the tiled one in its best width and cluster size (graph replays, cold
# weights). Only shapes on which the two are at least 6 % apart.
DECODE_SIZES = [
    (1, 1024, 2048, 4.1, 4.7), (1, 2048, 2048, 4.5, 5.3), (1, 768, 3072, 4.2, 4.9), (1, 7168, 7168, 14.7, 13.0),
    (1, 256, 7168, 6.2, 5.1), (8, 1536, 2560, 4.7, 5.5), (8, 12288, 5120, 18.0, 14.9), (16, 1536, 1536, 4.1, 4.6),
    (16, 2560, 2048, 4.7, 5.5), (16, 4096, 1024, 5.3, 4.1), (16, 12288, 4096, 15.0, 13.2),
    (16, 3072, 7168, 10.5, 8.9), (1, 16384, 2048, 9.9, 9.1), (16, 12288, 1024, 6.6, 6.2), (17, 1024, 2048, 4.4, 4.9),
    (17, 1536, 2048, 4.5, 5.3), (17, 7040, 1024, 5.7, 4.9), (17, 9216, 3072, 10.0, 8.5),
    (17, 8192, 7168, 18.4, 14.3), (17, 4096, 1536, 5.7, 4.8), (32, 1536, 3072, 5.2, 6.0), (32, 1024, 2048, 4.4, 5.0),
    (32, 7040, 2048, 7.7, 6.6), (32, 8192, 5120, 13.6, 11.9), (32, 7168, 5120, 12.3, 11.5),
    (32, 4096, 7168, 11.2, 10.4), (33, 2048, 1536, 5.0, 4.7), (33, 8192, 4096, 13.4, 10.2),
    (48, 512, 1536, 4.8, 4.2), (64, 1024, 7168, 8.8, 7.1), (64, 8192, 4096, 14.1, 10.2),
    (64, 8192, 7168, 21.1, 15.2), (64, 12288, 4096, 28.3, 13.0), (64, 1536, 3072, 6.6, 6.2)
]


@pytest.mark.parametrize("M,N,K,decode_us,tiled_us", DECODE_SIZES)
def test_decode_sizes_take_the_kernel_that_measured_faster(M, N, K, decode_us, tiled_us):
    assert _gemm_plan(M, N, K)["kernel"] == (DECODE if decode_us < tiled_us else TILED)


@pytest.mark.parametrize("M", [1, 16, 17, 32, 33, 64, 65, 129, 512, 777, 2200])
def test_automatic_plans_cover_k_with_resident_clusters(M):
    """Every CTA of a cluster has K blocks, and all clusters are on the GPU at once."""
    kernels = set()
    for N in list(range(16, 1040, 48)) + list(range(1040, 24577, 1296)):
        for K in list(range(128, 1281, 128)) + list(range(1536, 16385, 896)):
            plan = _gemm_plan(M, N, K)
            kernels.add(plan["kernel"])
            if plan["kernel"] == TILED:
                tiles = -(-M // 128) * -(-N // plan["block_n"])
                assert (plan["splits"] - 1) * plan["kbps"] < K // 128 <= plan["splits"] * plan["kbps"]
                assert plan["splits"] <= (4 if plan["block_n"] == 256 else 8)
                assert plan["ctas"] == (tiles * plan["splits"] if plan["splits"] > 1 else min(tiles, SMS)) <= SMS
    assert TILED in kernels and (M > 32 or DECODE in kernels) and (M <= 64 or DECODE not in kernels)
