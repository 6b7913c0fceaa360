"""The mat-vec kernels at row lengths around their cuts: rows of whole 64-weight chunks that are not a power of two (groups of
lanes with and without idle ones, more groups than warps, rows longer than 32 chunks), row counts that end inside a step, both
seed formats; gathers, gate+up with the router in front, dense calls of 1..8 rows.  The oracle's double-precision sums and the
bounds of the other mat-vec tests (one bf16 unit plus 64 x 1.2e-7 x sum|w x|)."""
import numpy as np
import pytest

from oracle import binding as B

pytestmark = pytest.mark.gpu
F32B = 64 * 1.2e-7


def matrices(p, n, R, K, seed):
    from nanoseedlm_b200 import kernels
    if p == 4:
        mats = [B.Matrix(R, K, seed + s, eb=-20 - s % 3) for s in range(n)]
        return [B.decode_rows_f32(m).astype(np.float64) for m in mats], kernels.SeedWeight.from_matrices(mats)
    mats = [B.Matrix3(R, K, seed + s, eb=-20 - s % 3) for s in range(n)]
    return [B.decode3_rows_f32(m).astype(np.float64) for m in mats], kernels.SeedWeight3(mats)


def check(got, W, x, extra=1.0):
    ref = B.bfr((W @ x).astype(np.float32)).astype(np.float64)
    assert (np.abs(got - ref) <= np.abs(ref) / 128 + extra * F32B * (np.abs(W) @ np.abs(x)) + 1e-30).all()


@pytest.mark.parametrize("p", [4, 3])
@pytest.mark.parametrize("K,R", [(64 * 3, 5), (64 * 7, 66), (64 * 11, 37), (64 * 24, 130), (64 * 33, 9), (64 * 45, 33), (64 * 96, 21)])
def test_any_number_of_chunks(p, K, R):
    from nanoseedlm_b200 import kernels
    W, w = matrices(p, 3, R, K, K + R)
    U, u = matrices(p, 3, R, K, 7 * K + R)
    x = B.bfr(np.random.default_rng(K).standard_normal((8, K)).astype(np.float32))
    sel = np.array([2, 0, 1, 1, 2, 0, 1], np.int32)
    mv_sel, mv_gu, mv = (kernels.kt_mv_sel, kernels.kt_mv_gu, kernels.kt_mv) if p == 4 else (kernels.kt_mv3_sel, kernels.kt_mv3_gu, kernels.kt_mv3)
    y, a = mv_sel(w, sel, 1, x[:7]), mv_gu(w, u, sel, 1, x[:7])
    for i, e in enumerate(sel):
        check(y[i], W[e], x[i].astype(np.float64))
        g, h = (B.bfr((M[e] @ x[i].astype(np.float64)).astype(np.float32)).astype(np.float64) for M in (W, U))
        silu = g / (1 + np.exp(-g))
        assert (np.abs(a[i] - silu * h) <= (np.abs(h) * (np.abs(g) + 1) + np.abs(silu * h)) / 64 + 1e-6).all()
    assert np.array_equal(mv_sel(w, sel[3:4], 1, x[3:4])[0], y[3])      # a pair alone: the same bits
    first = None
    for T in (1, 2, 5, 8):
        d = mv(w, x[:T], T)
        for t in range(T):
            check(d[t], W[0], x[t].astype(np.float64))
        first = d[0] if first is None else first
        assert np.array_equal(d[0], first)


@pytest.mark.parametrize("K,R,T", [(64 * 24, 88, 5), (64 * 6, 64, 8), (64 * 45, 40, 1)])
def test_router_in_front_at_any_number_of_chunks(K, R, T):
    from nanoseedlm_b200 import kernels
    E, k = 20, 3
    _, w = matrices(4, E, R, K, 11)
    _, u = matrices(4, E, R, K, 500)
    rng = np.random.default_rng(R)
    x = B.bfr(rng.standard_normal((T, K)).astype(np.float32))
    logits = rng.standard_normal((T, E)).astype(np.float32)
    a, ind, wt = kernels.kt_mv_gu_routed(w, u, logits, k, x)
    rind, rwt = B.route(logits, k)
    assert np.array_equal(ind, rind) and np.allclose(wt, rwt, rtol=1e-6)
    assert np.array_equal(a, kernels.kt_mv_gu(w, u, ind.ravel(), k, x))


@pytest.mark.parametrize("d,ff,E,k,T", [(256, 256, 28, 6, 8), (256, 256, 29, 6, 8), (256, 320, 8, 6, 8), (192, 512, 8, 6, 8), (2048, 64, 8, 8, 7)])
def test_decode_rows_whose_pairs_meet(d, ff, E, k, T):
    """A layer's decode rows either side of the line where pairs that meet on an expert share its expansion (48 pairs, 28 or 29 experts), and
    with one of the two products outside the grouped kernel's widths: every row has the bits it has alone."""
    from nanoseedlm_b200 import moe
    m = moe.Moe(moe.DeviceLayer.from_host(moe.HostLayer(B, d, ff, E, seed=d + E)), k, T)
    rng = np.random.default_rng(E)
    x = B.bfr(rng.standard_normal((T, d)).astype(np.float32))
    logits = rng.standard_normal((T, E)).astype(np.float32)
    out, ind = m.forward_host(x, logits)
    assert np.array_equal(ind, B.route(logits, k)[0])
    for t in range(T):
        assert np.array_equal(out[t], m.forward_host(x[t:t + 1], logits[t:t + 1])[0][0]), t
    m.close()


@pytest.mark.parametrize("K,R", [(64 * 3, 40), (64 * 11, 37), (64 * 24, 130), (64 * 45, 33)])
@pytest.mark.parametrize("by", [2, 8])
def test_p3_gathers_from_any_address(K, R, by):
    """Slices of a device table whose streams start off the 16-byte grid, between ones that do not: the aligned streams' bits."""
    import torch
    from nanoseedlm_b200 import kernels, lib as L
    _, w = matrices(3, 3, R, K, K + R)
    _, u = matrices(3, 3, R, K, 7 * K + R)
    x = B.bfr(np.random.default_rng(K).standard_normal((7, K)).astype(np.float32))
    sel = np.array([2, 0, 1, 1, 2, 0, 1], np.int32)
    ref = kernels.kt_mv3_sel(w, sel, 1, x), kernels.kt_mv3_gu(w, u, sel, 1, x), kernels.kt_mv3(w, x[:5], 5, s=1)
    for m, odd in ((w, (1,)), (u, (0, 1))):
        arr = (L.WSlice * 3)()
        for s in range(3):
            arr[s] = m.slice(s)
            for i, t in enumerate((m.seeds, m.nibs)):
                if s in odd:
                    buf = torch.empty(t[s].numel() + 8, dtype=t.dtype, device="cuda")
                    buf[by // 2:by // 2 + t[s].numel()] = t[s]
                    arr[s].p[i] = buf.data_ptr() + by
                    m.__dict__.setdefault("keep", []).append(buf)
        m.table = torch.frombuffer(bytearray(bytes(arr)), dtype=torch.uint8).cuda()
        m.slice = lambda s, arr=arr: arr[s]
    assert np.array_equal(kernels.kt_mv3_sel(w, sel, 1, x), ref[0])
    assert np.array_equal(kernels.kt_mv3_gu(w, u, sel, 1, x), ref[1])
    for t in range(5):
        assert (np.abs(kernels.kt_mv3(w, x[:5], 5, s=1)[t] - ref[2][t]) <= np.abs(ref[2][t]) / 64 + 1e-4 * np.abs(ref[2]).max()).all()


@pytest.mark.parametrize("p", [4, 3])
@pytest.mark.parametrize("R", [1, 31, 33, 64, 65, 130])
def test_rows_of_one_chunk(p, R):
    """K = 64: a lane is a row and keeps both of an item's sums; rows either side of one and two row steps."""
    test_any_number_of_chunks(p, 64, R)


@pytest.mark.parametrize("p", [4, 3])
@pytest.mark.parametrize("K,R", [(512, 40), (2048, 296), (2048, 593), (4096, 1184), (64 * 45, 1185), (64 * 200, 30), (64 * 300, 30)])
def test_dense_rows_of_small_matrices(p, K, R):
    """Matrices whose row steps leave warps over: 2 .. 8 rows of inputs in one group, in several, or (long rows) in two launches; every
    row has the bits it has alone, with the residual added too."""
    from nanoseedlm_b200 import kernels
    W, w = matrices(p, 1, R, K, K + R)
    mv = kernels.kt_mv if p == 4 else kernels.kt_mv3
    rng = np.random.default_rng(R)
    x, y0 = (B.bfr(rng.standard_normal((8, n)).astype(np.float32)) for n in (K, R))
    alone = [mv(w, x[t:t + 1], 1, add=1, y0=y0[t:t + 1])[0] for t in range(8)]
    check(mv(w, x[:1], 1)[0], W[0], x[0].astype(np.float64))
    for T in range(2, 9):
        d = mv(w, x[:T], T, add=1, y0=y0[:T])
        for t in range(T):
            assert np.array_equal(d[t], alone[t]), (T, t)


@pytest.mark.parametrize("p", [4, 3])
@pytest.mark.parametrize("K,R", [(128, 592), (128, 577), (128, 15)])
def test_gathers_either_side_of_one_row_step_an_item(p, K, R):
    """64 and 65 pairs of 37 row steps are one item a warp of 148 multiprocessors, and one more pair: items of one row step and of two (the last
    one single), with the same bits."""
    from nanoseedlm_b200 import kernels
    W, w = matrices(p, 3, R, K, K + R)
    x = B.bfr(np.random.default_rng(R).standard_normal((66, K)).astype(np.float32))
    sel = (np.arange(66) * 7 % 3).astype(np.int32)
    mv_sel = kernels.kt_mv_sel if p == 4 else kernels.kt_mv3_sel
    y = {P: mv_sel(w, sel[:P], 1, x[:P]) for P in (1, 2, 63, 64, 65, 66)}
    for P, v in y.items():
        assert np.array_equal(v, y[66][:P]), P
    for i in (0, 1, 37, 63, 64, 65):
        check(y[66][i], W[sel[i]], x[i].astype(np.float64))
