"""Edges of the kernels' tiles and of the dispatch's ranges, against the CPU oracle or a plain product."""
import numpy as np
import pytest

import oracle_lib as O
from moe_cases import Exl3Case, Exl3K2Case, Mxfp4Case, Nvfp4Case, max_err_over_rms, rel_l2
from test_parity_shapes_gpu import _shared_ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [(12, 13, 16, 17), (31, 32, 33, 1), (96, 97, 128, 129), (160, 161, 192, 193), (256, 257, 384, 385),
                                  (161,) + (17,) * 16])   # the last: one tile in sixteen more lets all tiles be narrow
@pytest.mark.parametrize("cls,limit", [(Exl3Case, 10.0), (Exl3K2Case, 10.0), (Mxfp4Case, 0.0), (Nvfp4Case, 10.0)])
def test_rows_of_an_expert_around_the_lanes_tiles(cls, limit, rows):
    """Row counts on both sides of the lane choice and of the tensor-core lane's row tiles, three weight blocks of 128 wide
    (an odd count: the last pass of the pair is short)."""
    fp4 = cls in (Mxfp4Case, Nvfp4Case)
    case = cls(768, 384, len(rows), 1, seed=21, shared=False, scoring=O.SCORE_SIGMOID, max_tokens=1300, routed_scale=1.0, limit=limit,
               chain=fp4)
    try:
        ids = np.random.default_rng(rows[0]).permutation(np.repeat(np.arange(len(rows)), rows)).astype(np.int32)[:, None]
        x, _ = case.inputs(ids.size, seed=40)
        w = np.full(ids.shape, 0.75, np.float32)
        y = case.gpu_experts(x, ids, w)
        assert case.status() == 0
        ref = case.cpu_layer(x, ids, w)
        for e in range(len(rows)):   # every expert by itself: one wrong tile is not averaged away
            m = ids[:, 0] == e
            assert rel_l2(y[m], ref[m]) < 1e-2, (e, rows[e])
    finally:
        case.close()


@pytest.mark.parametrize("E", [16, 64, 120, 256, 288])
def test_router_logits_around_the_change_of_kernel(E):
    """Few tokens (rows staged), tiles of 8 x 8 and, for 256 experts, 64 and 65 (tiles, tensor-core product); expert counts
    that leave a tile half empty."""
    import torch
    case = Exl3Case(640, 256, E, 4, seed=2, shared=False, max_tokens=1030, experts_to_load=[])
    try:
        wg = O.f32_to_bf16_bits((np.random.default_rng(5).standard_normal((E, 640)) * 0.05).astype(np.float32))
        case.moe.set_router_weight(0, wg.ctypes.data)
        wf = O.bf16_bits_to_f32(wg).astype(np.float64)
        for T in (1, 16, 17, 32, 33, 64, 65, 193, 1025):
            x, _ = case.inputs(T, seed=70 + T)
            lg = torch.full((T + 1, E), 7.0, dtype=torch.float32, device=case.dev)
            case.moe.logits(0, case.to_dev_bf16(x).data_ptr(), T, lg.data_ptr(), None)
            torch.cuda.synchronize()
            got = lg.cpu().numpy()
            assert np.allclose(got[:T], x.astype(np.float64) @ wf.T, rtol=2e-5, atol=1e-4), T
            assert (got[T] == 7.0).all()        # the padding is not stored
        assert case.status() == 0
    finally:
        case.close()


@pytest.mark.parametrize("H,I", [(512, 256), (1280, 768)])
def test_shared_expert_products_of_every_cluster_size(H, I):
    """The skinny kernel's token tiles, then the tensor-core products' tiles and clusters."""
    case = Exl3Case(H, I, 2, 1, seed=11, shared=True, max_tokens=1030)
    try:
        for T in (16, 17, 32, 33, 65, 96, 97, 129, 192, 193, 257, 1025):
            x, _ = case.inputs(T, seed=T)
            y = case.gpu_experts(x, np.zeros((T, 1), np.int32), np.zeros((T, 1), np.float32))
            assert case.status() == 0
            assert rel_l2(y, _shared_ref(x, case.shared, case.limit)) < 4e-3, T
    finally:
        case.close()


@pytest.mark.parametrize("cls,chain", [(Exl3Case, False), (Nvfp4Case, True)])
@pytest.mark.parametrize("H,k", [(384, 1), (512, 3), (1152, 9), (2176, 8)])
def test_combine_of_ragged_widths_and_counts(cls, chain, H, k):
    """Columns that do not fill a block, and expert counts around the eight rows a thread holds in flight."""
    case = cls(H, 256, 12, k, seed=5, shared=True, max_tokens=16, limit=10.0, chain=chain)
    try:
        x, logits = case.inputs(5, seed=3)
        ids, w = case.cpu_route(logits)
        y = case.gpu_forward(x, logits)
        assert case.status() == 0
        assert rel_l2(y, case.cpu_layer(x, ids, w)) < 1e-2
    finally:
        case.close()


@pytest.mark.parametrize("E", [1, 33, 256, 1024])
def test_dispatch_around_its_warps_and_blocks(E):
    import torch
    case = Exl3Case(128, 128, E, 1, seed=1, shared=False, max_tokens=17 * 1024 + 1, experts_to_load=[])
    try:
        rng = np.random.default_rng(E)
        for n in (1, 31, 32, 33, 1023, 1024, 1025, 2047, 2048, 2049, 17 * 1024 + 1):
            for slot in (rng.integers(0, E, n).astype(np.int32), np.full(n, E - 1, np.int32)):
                d = torch.from_numpy(slot).cuda()
                order = torch.full((n,), -1, dtype=torch.int32, device="cuda")
                offs = torch.full((E + 1,), -1, dtype=torch.int32, device="cuda")
                case.moe.sort_rows(d.data_ptr(), n, E, order.data_ptr(), offs.data_ptr(), None)
                torch.cuda.synchronize()
                assert (order.cpu().numpy() == np.argsort(slot, kind="stable")).all(), n
                assert (offs.cpu().numpy()[1:] == np.cumsum(np.bincount(slot, minlength=E))).all(), n
        assert case.status() == 0
    finally:
        case.close()


@pytest.mark.parametrize("E,k", [(8, 8), (31, 4), (256, 8), (288, 8)])
@pytest.mark.parametrize("scoring", [O.SCORE_SQRTSOFTPLUS, O.SCORE_SIGMOID, O.SCORE_SOFTMAX])
def test_front_of_a_small_call_routes_as_the_router_alone(scoring, E, k):
    """The fused front (one warp or one CTA per token) and the router kernel give the same layer, 1 to 17 tokens."""
    case = Exl3Case(256, 128, E, k, seed=6, shared=False, scoring=scoring, max_tokens=32)
    try:
        for T in (1, 2, 16, 17):
            x, logits = case.inputs(T, seed=T)
            ids, w = case.gpu_route(logits)
            assert (ids == case.cpu_route(logits)[0]).all()
            assert (case.gpu_forward(x, logits) == case.gpu_experts(x, ids, w)).all(), T
        assert case.status() == 0
    finally:
        case.close()


@pytest.mark.parametrize("cls,scales", [(Mxfp4Case, [0, 1, 109, 126, 127, 128, 130]), (Nvfp4Case, [0, 1, 7, 8, 9, 119, 126])])
def test_fp4_scale_bytes_at_the_ends_of_their_range(cls, scales):
    """Zero, subnormal and the largest scales through the streaming kernels' conversions."""
    nv = cls is Nvfp4Case
    case = cls(512, 256, 2, 1, seed=4, shared=False, scoring=O.SCORE_SIGMOID, max_tokens=16, routed_scale=1.0,
               limit=10.0 if nv else 0.0, chain=True)
    try:
        rec = case.records[0].copy()
        off = (O.nvfp4_record_bytes if nv else O.mxfp4_record_bytes)(512, 256)[1]
        n = 512 * 256 // (16 if nv else 32)
        s = off[1]                                # the gate projection's scales
        rec[s:s + n] = np.resize(np.array(scales, np.uint8), n)
        case.records[0] = rec
        case.moe.load_expert(0, 0, rec.ctypes.data, rec.size, on_device=False)
        for T in (1, 7, 16):
            x, _ = case.inputs(T, seed=T)
            ids, w = np.zeros((T, 1), np.int32), np.ones((T, 1), np.float32)
            y = case.gpu_experts(x, ids, w)
            assert case.status() == 0 and np.isfinite(y).all()
            assert rel_l2(y, case.cpu_layer(x, ids, w)) < 1e-2, T
    finally:
        case.close()


@pytest.mark.parametrize("H,I", [(1280, 768), (4096, 2048)])
def test_dense_products_of_a_row_do_not_depend_on_the_batch(H, I):
    """A row of the shared expert and of the router's logits has the same bits in every call of 65 to 256 tokens, whatever
    tiles and clusters serve it (5 and 3, 9 and 8 parts of the sums; 5 and 16 for the logits); larger calls split into fewer
    parts and are checked against the plain product."""
    import torch
    case = Exl3Case(H, I, 256, 1, seed=11, shared=True, max_tokens=1030, experts_to_load=[0, 1])
    try:
        x, _ = case.inputs(1025, seed=5)
        ref = _shared_ref(x, case.shared, case.limit)
        wg = O.f32_to_bf16_bits((np.random.default_rng(5).standard_normal((256, H)) * H ** -0.5).astype(np.float32))
        case.moe.set_router_weight(0, wg.ctypes.data)
        lref = x.astype(np.float64) @ O.bf16_bits_to_f32(wg).astype(np.float64).T
        first = None
        for T in (65, 70, 96, 97, 128, 129, 160, 161, 192, 193, 200, 256, 257, 300, 512, 513, 768, 769, 1024, 1025):
            y = case.gpu_experts(x[:T], np.zeros((T, 1), np.int32), np.zeros((T, 1), np.float32))
            lg = torch.empty((T, 256), dtype=torch.float32, device=case.dev)
            case.moe.logits(0, case.to_dev_bf16(x[:T]).data_ptr(), T, lg.data_ptr(), None)
            torch.cuda.synchronize()
            got = lg.cpu().numpy()
            assert case.status() == 0
            assert rel_l2(y, ref[:T]) < 4e-3, T
            assert rel_l2(got, lref[:T]) < 5e-7, T      # 20 sums in f32 per part and 16 parts: a random walk of 36 roundings of 2^-24 is 3.6e-7
            if T <= 256:
                first = (y[:65], got[:65]) if first is None else first
                assert (y[:65] == first[0]).all() and (got[:65] == first[1]).all(), T
    finally:
        case.close()


@pytest.mark.parametrize("E,H", [(256, 4096), (252, 1152), (60, 640), (288, 2176)])
def test_router_logits_keep_their_f32_sums(E, H):
    """Up to 64 tokens, and at any count when the experts do not fill the tensor-core product's blocks, a token's logits are
    the bits of a call of that token alone, and off a 64-bit product by no more than f32 sums of H / 128 terms per lane."""
    import torch
    case = Exl3Case(H, 128, E, 4, seed=2, shared=False, max_tokens=1030, experts_to_load=[])
    try:
        wg = O.f32_to_bf16_bits((np.random.default_rng(5).standard_normal((E, H)) * H ** -0.5).astype(np.float32))
        case.moe.set_router_weight(0, wg.ctypes.data)
        x, _ = case.inputs(1025, seed=7)
        xd = case.to_dev_bf16(x)
        ref = x.astype(np.float64) @ O.bf16_bits_to_f32(wg).astype(np.float64).T

        def logits(t0, T):
            lg = torch.full((T + 1, E), 7.0, dtype=torch.float32, device=case.dev)
            case.moe.logits(0, xd.data_ptr() + t0 * H * 2, T, lg.data_ptr(), None)
            torch.cuda.synchronize()
            assert (lg[T] == 7.0).all()
            return lg[:T].cpu().numpy()
        one = np.concatenate([logits(t, 1) for t in range(80)])
        for T in (4, 5, 8, 9, 16, 17, 25, 31, 64) + (() if E % 256 == 0 else (65, 200, 1025)):
            got = logits(0, T)
            assert (got[:80] == one[:T]).all(), T
            # a lane's H / 128 sums, the butterfly's 5 and the fold's 3, as a random walk of roundings of 2^-24
            assert rel_l2(got, ref[:T]) < 2.0 ** -24 * (H / 128 + 8) ** 0.5, T
        assert case.status() == 0
    finally:
        case.close()


def test_router_logits_into_a_buffer_of_four_byte_alignment():
    """Logits need 4-byte alignment alone, at every count of tokens (row kernel, tiles, the tensor-core product with and
    without a cluster): the same values as in an aligned buffer, and nothing beside them.  Less alignment, or rows of x off
    16 bytes, is refused by name."""
    import torch
    case = Exl3Case(4096, 256, 256, 4, seed=2, shared=False, max_tokens=2400, experts_to_load=[])
    try:
        wg = O.f32_to_bf16_bits((np.random.default_rng(5).standard_normal((256, 4096)) * 4096 ** -0.5).astype(np.float32))
        case.moe.set_router_weight(0, wg.ctypes.data)
        x, _ = case.inputs(2400, seed=7)
        xd = case.to_dev_bf16(x)
        for T in (1, 17, 65, 200, 600, 2400):
            a = torch.empty((T, 256), dtype=torch.float32, device=case.dev)
            b = torch.full((T * 256 + 5,), 7.0, dtype=torch.float32, device=case.dev)
            case.moe.logits(0, xd.data_ptr(), T, a.data_ptr(), None)
            for off in (1, 2, 3):
                b.fill_(7.0)
                case.moe.logits(0, xd.data_ptr(), T, b.data_ptr() + 4 * off, None)
                torch.cuda.synchronize()
                assert torch.equal(b[off:off + T * 256], a.view(-1)), (T, off)
                assert (b[:off] == 7.0).all() and (b[off + T * 256:] == 7.0).all(), (T, off)
        for dx, dl, name in ((2, 0, "x_dev"), (8, 0, "x_dev"), (0, 2, "logits_dev")):
            with pytest.raises(case.pkg.MlxsError, match=name):
                case.moe.logits(0, xd.data_ptr() + dx, 70, b.data_ptr() + dl, None)
        assert case.status() == 0
    finally:
        case.close()


@pytest.mark.parametrize("scale", [253, 254, 255])
def test_mxfp4_scale_bytes_beyond_f32(scale):
    """Block scales whose products leave f32: the gate saturates at the activation's limit, byte 255 too (2^128, an infinity,
    and no NaN), in every form of the streaming kernel; with 20 rows an expert of such scales still streams."""
    H, I = 512, 256
    case = Mxfp4Case(H, I, 2, 1, seed=4, shared=False, scoring=O.SCORE_SIGMOID, max_tokens=32, routed_scale=1.0, limit=10.0, chain=True)
    try:
        off = O.mxfp4_record_bytes(H, I)[1]
        rec = case.records[0].copy()
        rec[off[0]:off[0] + H * I // 2] = 0x77         # the gate projection: 6 everywhere
        rec[off[1]:off[1] + H * I // 32] = scale
        case.records[0] = rec
        case.moe.load_expert(0, 0, rec.ctypes.data, rec.size, on_device=False)
        for T in (1, 7, 9, 16, 20):
            x, _ = case.inputs(T, seed=T)
            x = np.abs(x) + 0.125
            x = O.bf16_bits_to_f32(O.f32_to_bf16_bits(x.astype(np.float32)))
            ids, w = np.zeros((T, 1), np.int32), np.ones((T, 1), np.float32)
            y = case.gpu_experts(x, ids, w)
            assert case.status() == 0 and np.isfinite(y).all(), T
            assert rel_l2(y, case.cpu_layer(x, ids, w)) < 1e-2, T
    finally:
        case.close()


FRONT_SCRIPT = r"""
import sys
import numpy as np
sys.path.insert(0, "tests")
import oracle_lib as O
from moe_cases import Exl3Case
E, k, counts = int(sys.argv[1]), int(sys.argv[2]), [int(t) for t in sys.argv[3].split(",")]
case = Exl3Case(256, 128, E, k, seed=6, shared=False, scoring=O.SCORE_SOFTMAX, max_tokens=256)
wg = O.f32_to_bf16_bits((np.random.default_rng(5).standard_normal((E, 256)) / 16).astype(np.float32))
case.moe.set_router_weight(0, wg.ctypes.data)
case.moe.profile_enable(True)
for T in counts:
    x, logits = case.inputs(T, seed=T)
    case.moe.profile_read()
    y = case.gpu_forward(x, logits)
    fused = case.moe.profile_read()["dispatch"][1] == 0
    assert fused == (T * k <= 2048), T
    ids, w = case.gpu_route(logits)
    assert (ids == case.cpu_route(logits)[0]).all(), T
    assert (y == case.gpu_experts(x, ids, w)).all(), T
    assert case.status() == 0
print("ok")
"""


@pytest.mark.parametrize("E,k,counts", [(256, 8, "164,165,166,200,256,1"), (256, 16, "128,129,1"), (1024, 8, "64,256,1"), (1024, 64, "32,1")])
def test_front_of_more_tokens_than_shared_memory_holds_scores_of(E, k, counts):
    """With the front's limit raised (in a process of its own: the limit is read once), up to 2048 assignments start with the
    fused kernel whatever the experts, and a call that does not leaves it to the calls after it."""
    import os
    import subprocess
    import sys
    from pathlib import Path
    r = subprocess.run([sys.executable, "-c", FRONT_SCRIPT, str(E), str(k), counts], cwd=Path(__file__).resolve().parent.parent,
                       env=dict(os.environ, MLXS_FRONT_MAX="256"), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "ok" in r.stdout, r.stderr[-2000:]


@pytest.mark.parametrize("cls,E", [(Exl3Case, 256), (Exl3Case, 40), (Mxfp4Case, 256), (Nvfp4Case, 24)])
def test_few_rows_are_sorted_as_many(cls, E):
    """Up to 32 rows a thread per row finds its place, above that the scan does: the same permutation, and the rows of the
    tokens that both calls hold are the same bits (a chunk of rows per expert; more in the next test)."""
    import torch
    fp4 = cls is not Exl3Case
    case = cls(512, 256, E, 8, seed=4, shared=False, scoring=O.SCORE_SIGMOID, max_tokens=64, routed_scale=1.0, chain=fp4)
    try:
        rng = np.random.default_rng(E)
        for n in (1, 4, 8, 31, 32, 33):
            slot = rng.integers(0, E, n).astype(np.int32)
            d = torch.from_numpy(slot).cuda()
            order = torch.full((n,), -1, dtype=torch.int32, device="cuda")
            offs = torch.full((E + 1,), -1, dtype=torch.int32, device="cuda")
            case.moe.sort_rows(d.data_ptr(), n, E, order.data_ptr(), offs.data_ptr(), None)
            torch.cuda.synchronize()
            assert (order.cpu().numpy() == np.argsort(slot, kind="stable")).all(), n
            assert (offs.cpu().numpy() == np.concatenate([[0], np.cumsum(np.bincount(slot, minlength=E))])).all(), n
        hot = min(E, 20)   # 17 tokens of 8 experts among 20: fewer than 13 rows each with these seeds, so all of them stream
        ids = np.stack([np.random.default_rng(100 + t).permutation(hot)[:8] for t in range(17)]).astype(np.int32)
        assert np.bincount(ids.ravel()).max() < 13
        x, _ = case.inputs(17, seed=3)
        w = np.full(ids.shape, 0.125, np.float32)
        many = case.gpu_experts(x, ids, w)
        for T in (1, 3, 4, 5):
            assert (case.gpu_experts(x[:T], ids[:T], w[:T]) == many[:T]).all(), T
        same = np.broadcast_to(ids[0], (4, 8)).copy()   # four tokens of the same experts
        wide = np.concatenate([same, ids[4:9]])
        assert (case.gpu_experts(x[:4], same, w[:4]) == case.gpu_experts(x[:9], wide, w[:9])[:4]).all()
        assert rel_l2(many, case.cpu_layer(x, ids, w)) < 1e-2
        assert case.status() == 0
    finally:
        case.close()


@pytest.mark.parametrize("cls,counts", [(Exl3Case, (12, 9, 5, 4, 1, 1)), (Exl3Case, (8, 12, 12)), (Exl3K2Case, (4, 11, 8, 9)), (Mxfp4Case, (16, 9, 5, 1, 1)),
                                        (Mxfp4Case, (8, 15, 9)), (Nvfp4Case, (1, 16, 8, 7))])
def test_experts_of_several_chunks_in_a_short_call(cls, counts):
    """32 rows, experts with up to three chunks of rows: the bits that the same rows have in a call of 37, whose sort is the scan."""
    fp4 = cls in (Mxfp4Case, Nvfp4Case)
    case = cls(512, 256, 8, 1, seed=6, shared=False, scoring=O.SCORE_SIGMOID, max_tokens=64, routed_scale=1.0, limit=10.0, chain=fp4)
    try:
        ids = np.random.default_rng(sum(counts[:2])).permutation(np.repeat(np.arange(len(counts)), counts)).astype(np.int32)
        assert ids.size == 32
        more = np.concatenate([ids, np.full(5, 7, np.int32)])[:, None]
        x, _ = case.inputs(37, seed=8)
        w = np.full(more.shape, 0.75, np.float32)
        few = case.gpu_experts(x[:32], more[:32], w[:32])
        assert (few == case.gpu_experts(x, more, w)[:32]).all()
        ref = case.cpu_layer(x[:32], more[:32], w[:32])
        for e in range(len(counts)):
            assert rel_l2(few[ids == e], ref[ids == e]) < 1e-2, e
        assert case.status() == 0
    finally:
        case.close()


@pytest.mark.parametrize("cls", [Exl3Case, Exl3K2Case, Mxfp4Case, Nvfp4Case])
@pytest.mark.parametrize("split", [32, 20, 17, 16])
def test_experts_of_several_groups_in_a_short_call(cls, split):
    """Four tokens that name an expert eight times over: up to 32 rows of one expert in the streaming lane, two groups of chunks
    (16 rows), against five tokens (40 rows, the scan)."""
    fp4 = cls in (Mxfp4Case, Nvfp4Case)
    case = cls(512, 256, 8, 8, seed=7, shared=False, scoring=O.SCORE_SIGMOID, max_tokens=64, routed_scale=1.0, limit=10.0, chain=fp4)
    try:
        ids = np.random.default_rng(split).permutation(np.repeat([2, 5], [split, 32 - split])).reshape(4, 8).astype(np.int32)
        more = np.concatenate([ids, np.arange(8, dtype=np.int32)[None] % 2 * 6])   # experts 0 and 6
        x, _ = case.inputs(5, seed=9)
        w = np.random.default_rng(1).random(more.shape).astype(np.float32)
        few = case.gpu_experts(x[:4], ids, w[:4])
        assert (few == case.gpu_experts(x, more, w)[:4]).all()
        assert rel_l2(few, case.cpu_layer(x[:4], ids, w[:4])) < 1e-2
        assert case.status() == 0
    finally:
        case.close()


@pytest.mark.parametrize("W", [1, 2, 3, 8])
def test_few_rows_into_few_bins(W):
    """The short sort with the bin counts that an exchange between ranks has."""
    import torch
    case = Exl3Case(128, 128, 8, 1, seed=1, shared=False, max_tokens=64, experts_to_load=[])
    try:
        rng = np.random.default_rng(W)
        for n in range(1, 34):
            slot = rng.integers(0, W, n).astype(np.int32)
            d = torch.from_numpy(slot).cuda()
            order = torch.full((n,), -1, dtype=torch.int32, device="cuda")
            offs = torch.full((W + 1,), -1, dtype=torch.int32, device="cuda")
            case.moe.sort_rows(d.data_ptr(), n, W, order.data_ptr(), offs.data_ptr(), None)
            torch.cuda.synchronize()
            assert (order.cpu().numpy() == np.argsort(slot, kind="stable")).all(), n
            assert (offs.cpu().numpy() == np.concatenate([[0], np.cumsum(np.bincount(slot, minlength=W))])).all(), n
        assert case.status() == 0
    finally:
        case.close()


@pytest.mark.parametrize("cls,E,H,shared", [(Exl3Case, 256, 1024, False), (Exl3Case, 256, 6144, False), (Exl3Case, 64, 7168, False), (Exl3Case, 9, 1664, False),
                                            (Exl3Case, 288, 512, False), (Exl3Case, 1024, 256, False), (Nvfp4Case, 24, 512, True), (Mxfp4Case, 136, 256, False),
                                            (Nvfp4Case, 300, 256, True)])
def test_layer_from_x_of_a_few_tokens(cls, E, H, shared):
    """From x the front's CTAs share out experts, tokens (beyond 256 experts in two passes, a CTA's experts in two or more
    rounds) and (beyond 6144 inputs) a row's vectors in more than one round: the layer is the one that the logits alone give, 1
    to 16 tokens.  The FP4 banks' rows are staged by quarters beside the shared expert, from the logits by sixteenths."""
    import torch
    case = cls(H, 128, E, 4, seed=2, shared=shared, scoring=O.SCORE_SIGMOID, max_tokens=32, chain=cls is not Exl3Case)
    try:
        wg = O.f32_to_bf16_bits((np.random.default_rng(5).standard_normal((E, H)) * H ** -0.5).astype(np.float32))
        case.moe.set_router_weight(0, wg.ctypes.data)
        for T in (1, 2, 3, 7, 8, 9, 15, 16):
            x, _ = case.inputs(T, seed=20 + T)
            xd = case.to_dev_bf16(x)
            lg = torch.empty((T, E), dtype=torch.float32, device=case.dev)
            case.moe.logits(0, xd.data_ptr(), T, lg.data_ptr(), None)
            y = torch.empty((T, H), dtype=torch.bfloat16, device=case.dev)
            case.moe.forward_x(0, xd.data_ptr(), T, y.data_ptr(), None)
            torch.cuda.synchronize()
            assert (y.float().cpu().numpy() == case.gpu_forward(x, lg.cpu().numpy())).all(), T
        assert case.status() == 0
    finally:
        case.close()


@pytest.mark.parametrize("cls", [Exl3Case, Exl3K2Case])
def test_records_of_four_byte_alignment_load_the_same_bank(cls):
    """The repack reads a record in words, at any address that they allow."""
    import torch
    case = cls(384, 256, 2, 1, seed=9, shared=False, max_tokens=32, experts_to_load=[0])
    try:
        rec = torch.from_numpy(np.concatenate([np.zeros(4, np.uint8), case.records[0]])).cuda()
        case.moe.load_expert(0, 1, rec.data_ptr() + 4, rec.numel() - 4, on_device=True)
        x, _ = case.inputs(5, seed=1)
        w = np.ones((5, 1), np.float32)
        a, b = (case.gpu_experts(x, np.full((5, 1), e, np.int32), w) for e in (0, 1))
        assert np.isfinite(a).all() and np.abs(a).max() > 0 and (a == b).all()
        assert case.status() == 0
    finally:
        case.close()
