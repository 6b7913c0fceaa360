"""The prompt GEMM's ways through a layer and a dense call at the sizes where they change: rows an expert either side of the kernel
that keeps weights in registers and of the one that shares an expansion between tiles (units of one, two and three tiles,
ragged ends, experts without rows), rows of weights that end inside a tile, inputs in both forms.  Layers are compared with the
mat-vec path on the same rows (which does not round the seed weights to bf16), dense calls with the decoded weights."""
import numpy as np
import pytest

from oracle import binding as B

pytestmark = pytest.mark.gpu
F32B = 64 * 1.2e-7


@pytest.mark.parametrize("d,ff,E,k,T,skew", [(256, 128, 40, 3, 50, 0.0),      # 4 rows an expert: weights in registers
                                             (320, 192, 8, 2, 60, 0.0),      # 15: one tile; rows of weights end inside a tile
                                             (256, 64, 5, 2, 233, 2.0),      # 93, some experts over 128, one with few
                                             (256, 64, 4, 2, 600, 0.0),      # 300: two and three tiles share an expansion
                                             (128, 64, 6, 3, 900, 3.0),      # up to 900 rows: several units an expert
                                             (192, 320, 3, 1, 387, 0.0),
                                             (320, 192, 100, 3, 190, 9.0),   # 5 rows an expert, some with over 32 and over 128; chunks that do not fill a step
                                             (64, 64, 60, 2, 100, 0.0),      # one chunk a row
                                             (576, 448, 30, 2, 80, 4.0),
                                             (256, 64, 96, 8, 1024, 0.0),    # 8192 pairs: grouped in one launch
                                             (256, 64, 96, 8, 1025, 0.0)])   # more: in two
def test_layer_against_the_mat_vec_path(d, ff, E, k, T, skew):
    from nanoseedlm_b200 import moe
    layer = moe.DeviceLayer.from_host(moe.HostLayer(B, d, ff, E, seed=d + T))
    m = moe.Moe(layer, k, T)
    rng = np.random.default_rng(T)
    x = B.bfr(rng.standard_normal((T, d)).astype(np.float32))
    logits = (rng.standard_normal((T, E)) - skew * np.arange(E) / E).astype(np.float32)
    out, ind = m.forward_host(x, logits)
    assert np.array_equal(ind, B.route(logits, k)[0])
    m.set_grouped_min_tokens(10 ** 6)
    ref, _ = m.forward_host(x, logits)
    err = np.linalg.norm(out - ref, axis=1) / np.linalg.norm(ref, axis=1)
    assert err.max() < 1.5e-2, (int(err.argmax()), float(err.max()))
    m.close()


@pytest.mark.parametrize("p", [4, 3])
@pytest.mark.parametrize("R,K,T", [(130, 192, 9), (40, 1088, 33), (257, 256, 64), (100, 448, 65), (384, 128, 129), (64, 64, 400), (72, 136, 300)])
@pytest.mark.parametrize("packed", [False, True])
def test_dense(p, R, K, T, packed):
    from nanoseedlm_b200 import kernels
    m = B.Matrix(R, K, R + K, eb=-21) if p == 4 else B.Matrix3(R, K, R + K, eb=-21)
    W = B.bfr(B.decode_rows_f32(m) if p == 4 else B.decode3_rows_f32(m)).astype(np.float64)
    w = kernels.SeedWeight.from_matrices([m]) if p == 4 else kernels.SeedWeight3([m])
    x = B.bfr(np.random.default_rng(K).standard_normal((T, K)).astype(np.float32))
    y = kernels.kt_mm(w, x, T, packed=packed)
    acc = x.astype(np.float64) @ W.T
    ref = B.bfr(acc.astype(np.float32)).astype(np.float64)
    assert (np.abs(y - ref) <= np.abs(ref) / 128 + F32B * (np.abs(x.astype(np.float64)) @ np.abs(W.T)) + 1e-30).all()
