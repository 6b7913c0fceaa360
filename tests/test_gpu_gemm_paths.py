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


def routed_layer(d, ff, counts, seed, scale=1.0):
    """A layer of len(counts) experts, top 1, whose expert e gets counts[e] rows in a shuffled order -> (the handle's output, the rows'
    experts, decoded bf16 weights per expert, inputs); everything on the device."""
    import torch
    from nanoseedlm_b200 import kernels, lib as L, moe
    E, T = len(counts), int(sum(counts))
    gen = torch.Generator(device="cuda").manual_seed(seed)
    layer = moe.DeviceLayer.random_on_device(d, ff, E, gen)
    m = moe.Moe(layer, 1, T)
    expert = torch.repeat_interleave(torch.arange(E, device="cuda"), torch.tensor(counts, device="cuda"))[torch.randperm(T, generator=gen, device="cuda")]
    x = (torch.randn((T, d), generator=gen, device="cuda") * scale).to(torch.bfloat16).float()
    logits = torch.zeros((T, E), device="cuda").scatter_(1, expert[:, None], 8.0)
    out = torch.full((T, d), float("nan"), device="cuda")
    m.forward_dev(x, logits, out)
    again = torch.empty_like(out)
    m.forward_dev(x, logits, again)
    kernels._done()      # (raises when a GEMM block gave up on a wait)
    assert torch.equal(out, again)
    m.close()

    def decoded(stack, R, K):      # all experts as one matrix: their streams follow one another
        w = L.WSlice()
        w.p[0], w.p[1], w.p[3], w.eb = stack.seeds.data_ptr(), stack.coefs.data_ptr(), stack.codes.data_ptr(), stack.eb[0]
        o = torch.empty((E, R, K), dtype=torch.bfloat16, device="cuda")
        L.load().nsl_decode_bf16(kernels._stream(), w, K, E * R, kernels._ptr(o), kernels._ptr(kernels.stream_table()))
        return o
    return out, expert, (decoded(layer.gate, ff, d), decoded(layer.up, ff, d), decoded(layer.down, d, ff)), x


def layer_reference(weights, expert, x):
    """The layer's rows with its rounding points, sums in double precision, and sum |w a| of every output."""
    import torch
    r = lambda t: t.float().to(torch.bfloat16).double()
    ref, mag = torch.empty_like(x, dtype=torch.float64), torch.empty_like(x, dtype=torch.float64)
    for e in range(weights[0].shape[0]):
        rows = (expert == e).nonzero()[:, 0]
        if not len(rows):
            continue
        wg, wu, wd = (w[e].double() for w in weights)
        xe = x[rows].double()
        g, u = r(xe @ wg.T), r(xe @ wu.T)
        a = r(r(g * r(1.0 / (1.0 + torch.exp(-g)))) * u)
        ref[rows], mag[rows] = r(a @ wd.T), a.abs() @ wd.abs().T
    return ref, mag


# Rows an expert: units of one to three tiles, at most and more than half of the accumulators (192 rows), full (384) and one beyond.
UNITS = [97, 130, 192, 193, 110, 250, 100, 384, 96, 385, 120, 60, 140, 192, 150, 0]


@pytest.mark.parametrize("d,ff,E", [(128, 256, 480), (256, 128, 480), (192, 320, 256), (448, 256, 256), (256, 448, 256), (320, 192, 256), (576, 512, 160)])
def test_many_units_a_block_that_share_expansions(d, ff, E):
    """Prompts whose experts' tiles share an expansion, several units a block, 2 .. 9 K steps a unit: a warpgroup has no, one or two
    steps of a unit, and results are read under the next one.  Every element: an activation can round the other way, so an
    output may differ by what it is to have all of its row's activations a bf16 unit off."""
    out, expert, weights, x = routed_layer(d, ff, [UNITS[e % len(UNITS)] for e in range(E)], d + ff)
    ref, mag = layer_reference(weights, expert, x)
    assert ((out.double() - ref).abs() <= ref.abs() / 128 + mag / 128 + 1e-30).all()


@pytest.mark.parametrize("d,ff,E,k", [(512, 256, 32, 4), (320, 192, 12, 3), (1000, 504, 16, 2)])
def test_a_prompt_row_has_the_same_bits_in_every_batch(d, ff, E, k):
    """1 .. 500 rows an expert, evenly and unevenly routed: the batch's size and routing choose units, loaders and shared expansions,
    never the order of a row's sums."""
    import torch
    from nanoseedlm_b200 import kernels, moe
    gen = torch.Generator(device="cuda").manual_seed(d)
    layer = moe.DeviceLayer.random_on_device(d, ff, E, gen)
    T = 500 * E // k
    m = moe.Moe(layer, k, T)
    x = torch.randn((T, d), generator=gen, device="cuda").to(torch.bfloat16).float()
    logits = torch.randn((T, E), generator=gen, device="cuda")
    logits[T // 2:] -= 12.0 * torch.arange(E, device="cuda") / E
    outs = {}
    for n in (9, 16, 33, 64, 65, 100, 6 * E // k, 97 * E // k, T):
        out = torch.empty((n, d), device="cuda")
        m.forward_dev(x[:n].contiguous(), logits[:n].contiguous(), out)
        outs[n] = out
    kernels._done()
    for n, out in outs.items():
        assert torch.equal(out, outs[T][:n]), n
    m.close()


def shifted(t, by):
    """The tensor's bytes `by` bytes into a fresh buffer -> (address, buffer)."""
    import torch
    raw = t.contiguous().view(torch.uint8).flatten()
    buf = torch.empty(raw.numel() + 16, dtype=torch.uint8, device="cuda")
    buf[by:by + raw.numel()] = raw
    return buf.data_ptr() + by, buf


@pytest.mark.parametrize("p", [4, 3])
@pytest.mark.parametrize("R,K,T", [(130, 192, 20), (130, 192, 64), (70, 1088, 70), (140, 96, 300), (33, 160, 65), (40, 72, 40)])
@pytest.mark.parametrize("by", [0, 2, 8])
def test_dense_streams_of_any_alignment(p, R, K, T, by):
    """K of whole chunks, of half chunks and of neither; streams on 16, on 8 and on 2 bytes (codes on 4, 2 and 1)."""
    import torch
    from nanoseedlm_b200 import kernels, lib as L
    m = B.Matrix(R, K, R + K, eb=-21) if p == 4 else B.Matrix3(R, K, R + K, eb=-21)
    W = B.bfr(B.decode_rows_f32(m) if p == 4 else B.decode3_rows_f32(m)).astype(np.float64)
    w0 = kernels.SeedWeight.from_matrices([m]) if p == 4 else kernels.SeedWeight3([m])
    keep = [shifted(w0.seeds, by), shifted(w0.coefs if p == 4 else w0.nibs, by)] + ([shifted(w0.codes, {0: 0, 2: 1, 8: 2}[by])] if p == 4 else [])
    w = w0.slice(0)
    w.p[0], w.p[1] = keep[0][0], keep[1][0]
    if p == 4:
        w.p[3] = keep[2][0]
    x = B.bfr(np.random.default_rng(K).standard_normal((T, K)).astype(np.float32))
    xd = kernels.dev(x)
    ref = x.astype(np.float64) @ W.T
    bound = F32B * (np.abs(x.astype(np.float64)) @ np.abs(W.T)) + 1e-30
    ref = B.bfr(ref.astype(np.float32)).astype(np.float64)
    for packed in (False, True):
        y = torch.full((T, R), float("nan"), device="cuda")
        xin = xd.to(torch.bfloat16) if packed else xd
        (L.load().kc_mm_packed if packed else L.load().kc_mm)(kernels._stream(), L.MF_SEED4P4 if p == 4 else L.MF_SEED4, w, K, R, kernels._ptr(xin), K,
                                                              kernels._ptr(y), R, T, 0, kernels._ptr(kernels.stream_table()))
        kernels._done()
        assert (np.abs(y.cpu().numpy() - ref) <= np.abs(ref) / 128 + bound).all()


@pytest.mark.parametrize("d,ff,T", [(256, 128, 100), (192, 320, 1200)])
def test_a_layer_whose_streams_lie_on_8_bytes(d, ff, T):
    """The slices of a device table are looked at by the kernels: the same bits from streams that are only 8-byte (codes 2-byte) aligned, in
    every second expert."""
    import ctypes as C
    import torch
    from nanoseedlm_b200 import kernels, lib as L, moe
    E, k = 6, 2
    gen = torch.Generator(device="cuda").manual_seed(d)
    layer = moe.DeviceLayer.random_on_device(d, ff, E, gen)
    x, logits = torch.randn((T, d), generator=gen, device="cuda").to(torch.bfloat16).float(), torch.randn((T, E), generator=gen, device="cuda")
    m = moe.Moe(layer, k, T)
    ref, out = torch.empty((T, d), device="cuda"), torch.empty((T, d), device="cuda")
    m.forward_dev(x, logits, ref)
    tables, keep = [], []
    for st in (layer.gate, layer.up, layer.down):
        arr = (L.WSlice * E)()
        for e in range(E):
            s = [shifted(t[e], by if e & 1 else 0) for t, by in ((st.seeds, 8), (st.coefs, 8), (st.codes, 2))]
            keep.append(s)
            arr[e].p[0], arr[e].p[1], arr[e].p[3], arr[e].eb = s[0][0], s[1][0], s[2][0], st.eb[e]
        tables.append(torch.frombuffer(bytearray(bytes(arr)), dtype=torch.uint8).cuda())
    m.lib.nsl_moe_set_layer(m.h, *(kernels._ptr(t) for t in tables))
    m.forward_dev(x, logits, out)
    kernels._done()
    assert torch.equal(out, ref)
    m.close()


@pytest.mark.parametrize("T", [36, 216])      # the GEMM's two forms of the gate + up product
def test_swiglu_over_the_range_of_gates(T):
    """Rows whose gates all lie at one value, from where the sigmoid is a subnormal bf16 number (below -87.3; e^-g overflows f32 below -88.7)
    to where it is 1.  A gate that rounds to the neighbouring bf16 value moves its own activation by up to e^0.5, one of 64: rows are
    compared by their norms."""
    import torch
    from nanoseedlm_b200 import kernels, lib as L, moe
    d, ff = 1024, 64
    gen = torch.Generator(device="cuda").manual_seed(T)
    layer = moe.DeviceLayer.random_on_device(d, ff, 1, gen)

    def decoded(stack, R, K):
        w = L.WSlice()
        w.p[0], w.p[1], w.p[3], w.eb = stack.seeds.data_ptr(), stack.coefs.data_ptr(), stack.codes.data_ptr(), stack.eb[0]
        o = torch.empty((1, R, K), dtype=torch.bfloat16, device="cuda")
        L.load().nsl_decode_bf16(kernels._stream(), w, K, R, kernels._ptr(o), kernels._ptr(kernels.stream_table()))
        return o
    weights = decoded(layer.gate, ff, d), decoded(layer.up, ff, d), decoded(layer.down, d, ff)
    gates = torch.tensor([-88.0, -87.75, -87.5, -87.25, -87.0, -80.0, -40.0, -8.0, -1.0, 1.0, 8.0, 100.0], device="cuda", dtype=torch.float64).repeat(T // 12)
    x = (gates[:, None] * (torch.linalg.pinv(weights[0][0].double()) @ torch.ones(ff, device="cuda", dtype=torch.float64))).to(torch.bfloat16).float()
    m = moe.Moe(layer, 1, T)
    out = torch.empty((T, d), device="cuda")
    m.forward_dev(x, torch.zeros((T, 1), device="cuda"), out)
    kernels._done()
    m.close()
    ref, _ = layer_reference(weights, torch.zeros(T, dtype=torch.long, device="cuda"), x)
    assert (ref.norm(dim=1) > 0).all()
    err = (out.double() - ref).norm(dim=1) / ref.norm(dim=1)
    assert (err < 0.25).all(), err[:12]


@pytest.mark.parametrize("xs", [0, 64, 184, 192, 200])
@pytest.mark.parametrize("T", [40, 70, 500])
def test_packed_rows_at_any_distance(xs, T):
    """Packed rows that repeat, overlap, follow one another or lie apart (a tensor map describes the last two)."""
    import torch
    from nanoseedlm_b200 import kernels, lib as L
    R, K = 150, 192
    m = B.Matrix(R, K, 5, eb=-21)
    w = kernels.SeedWeight.from_matrices([m])
    W = B.bfr(B.decode_rows_f32(m)).astype(np.float64)
    flat = B.bfr(np.random.default_rng(xs).standard_normal((T - 1) * xs + K).astype(np.float32))
    x = np.stack([flat[t * xs:t * xs + K] for t in range(T)]).astype(np.float64)
    xd, y = kernels.dev(flat).to(torch.bfloat16), torch.full((T, R), float("nan"), device="cuda")
    L.load().kc_mm_packed(kernels._stream(), L.MF_SEED4P4, w.slice(0), K, R, kernels._ptr(xd), xs, kernels._ptr(y), R, T, 0, kernels._ptr(kernels.stream_table()))
    kernels._done()
    ref = B.bfr((x @ W.T).astype(np.float32)).astype(np.float64)
    assert (np.abs(y.cpu().numpy() - ref) <= np.abs(ref) / 128 + F32B * (np.abs(x) @ np.abs(W.T)) + 1e-30).all()


def decoded_stack(stack, E):
    """A device stack's weights, exact and rounded to bf16 once: [E][R][K]."""
    import torch
    from nanoseedlm_b200 import kernels, lib as L
    w = L.WSlice()
    w.p[0], w.p[1], w.p[3], w.eb = stack.seeds.data_ptr(), stack.coefs.data_ptr(), stack.codes.data_ptr(), stack.eb[0]
    o = torch.empty((E, stack.R, stack.K), dtype=torch.bfloat16, device="cuda")
    L.load().nsl_decode_bf16(kernels._stream(), w, stack.K, E * stack.R, kernels._ptr(o), kernels._ptr(kernels.stream_table()))
    return o


def within(y, x, W):
    ref, mag = x.double() @ W.double().T, x.double().abs() @ W.double().abs().T
    return ((y.double() - ref).abs() <= ref.abs() / 128 + F32B * mag + 1e-30).all()


@pytest.mark.parametrize("K", [64, 128, 192, 256, 320, 448])
@pytest.mark.parametrize("packed", [False, True])
def test_grouped_tiles_of_every_size_many_units_a_block(K, packed):
    """Tiles of 1 .. 128 rows, either side of where the loaders' warps share out the K steps (40, 60) and of half of the accumulators, in no
    order, three to seven units a block; every element."""
    import torch
    from nanoseedlm_b200 import kernels, lib as L, moe
    counts = [1, 64, 128, 16, 17, 65, 40, 41, 48, 100, 49, 60, 61, 127, 32, 33, 8, 96, 80, 63, 112, 62, 24, 57, 56, 9]
    E, R, P = len(counts), 5210, sum(counts)
    gen = torch.Generator(device="cuda").manual_seed(K)
    st = moe.ExpertStack.random_on_device(E, R, K, gen)
    W = decoded_stack(st, E)
    sel = torch.repeat_interleave(torch.arange(E, device="cuda"), torch.tensor(counts, device="cuda"))
    perm = torch.randperm(P, generator=gen, device="cuda").int()      # pair perm[i] belongs to the i-th place's expert
    tiles = torch.zeros((E, 4), dtype=torch.int32)
    tiles[:, 0], tiles[:, 2] = torch.arange(E), torch.tensor(counts)
    tiles[1:, 1] = torch.tensor(counts).cumsum(0)[:-1]
    x = torch.randn((P, K), generator=gen, device="cuda").to(torch.bfloat16)
    xin, y, nt = (x if packed else x.float()), torch.full((P, R), float("nan"), device="cuda"), torch.tensor([E], dtype=torch.int32, device="cuda")
    tiles = tiles.cuda()
    f = L.load().kc_mm_grouped_packed if packed else L.load().kc_mm_grouped_dev
    f(kernels._stream(), L.MF_SEED4P4, kernels._ptr(st.table), K, R, kernels._ptr(xin), K, kernels._ptr(y), R, 1, kernels._ptr(perm), kernels._ptr(tiles),
      kernels._ptr(nt), E + 2, kernels._ptr(kernels.stream_table()))
    kernels._done()
    for e in range(E):
        rows = perm[sel == e].long()
        assert within(y[rows], x[rows].float(), W[e].float()), counts[e]


@pytest.mark.parametrize("R,K,T", [(75800, 64, 70), (75800, 192, 128), (75800, 256, 130), (115200, 320, 100), (40000, 448, 300), (40000, 128, 500)])
@pytest.mark.parametrize("packed", [False, True])
def test_dense_calls_of_many_units_a_block(R, K, T, packed):
    import torch
    from nanoseedlm_b200 import kernels, lib as L, moe
    gen = torch.Generator(device="cuda").manual_seed(T)
    st = moe.ExpertStack.random_on_device(1, R, K, gen)
    W = decoded_stack(st, 1)[0].float()
    w = L.WSlice()
    w.p[0], w.p[1], w.p[3], w.eb = st.seeds.data_ptr(), st.coefs.data_ptr(), st.codes.data_ptr(), st.eb[0]
    x = torch.randn((T, K), generator=gen, device="cuda").to(torch.bfloat16)
    xin, y = (x if packed else x.float()), torch.full((T, R), float("nan"), device="cuda")
    (L.load().kc_mm_packed if packed else L.load().kc_mm)(kernels._stream(), L.MF_SEED4P4, w, K, R, kernels._ptr(xin), K, kernels._ptr(y), R, T, 0,
                                                          kernels._ptr(kernels.stream_table()))
    kernels._done()
    assert within(y, x.float(), W)


@pytest.mark.parametrize("p", [4, 3])
@pytest.mark.parametrize("R,K", [(300, 256), (2048, 512), (130, 1088), (70, 96)])
@pytest.mark.parametrize("packed", [False, True])
def test_a_dense_row_has_the_same_bits_up_to_64_rows_and_from_65_on(p, R, K, packed):
    """Two kernels with their own orders of the sums; within each (and, where K is not a multiple of 64, over both ranges: one kernel) a row's
    bits do not depend on the number of rows."""
    from nanoseedlm_b200 import kernels
    m = B.Matrix(R, K, R + K, eb=-21) if p == 4 else B.Matrix3(R, K, R + K, eb=-21)
    w = kernels.SeedWeight.from_matrices([m]) if p == 4 else kernels.SeedWeight3([m])
    x = B.bfr(np.random.default_rng(K).standard_normal((700, K)).astype(np.float32))
    mm = lambda T: kernels.kt_mm(w, x[:T], T, packed=packed)
    few, many = mm(64), mm(700)
    for T in (1, 8, 9, 16, 17, 32, 33, 63):
        assert np.array_equal(mm(T), few[:T]), T
    for T in (65, 128, 129, 256, 257, 384, 385, 500):
        assert np.array_equal(mm(T), many[:T]), T
    if K % 64:
        assert np.array_equal(few, many[:64])


@pytest.mark.parametrize("p", [4, 3])
@pytest.mark.parametrize("R,K,T", [(130, 64, 65), (130, 128, 129), (257, 192, 257), (300, 1024, 128), (-1, 128, 100), (0, 128, 100), (1, 128, 100),
                                   (2048, 320, 1300), (2048, 64, 1409), (2050, 192, 2307), (1000, 128, 4100)])
def test_dense_f32_rows_have_the_bits_of_the_packed_ones(p, R, K, T):
    """Blocks of one unit with one, two or three tiles of rows, and (one tile) blocks of several: the same values meet in the same MMAs in
    the same order as with packed inputs, whatever the loaders."""
    import torch
    from nanoseedlm_b200 import kernels
    if R < 2: R += 128 * torch.cuda.get_device_properties(0).multi_processor_count      # just one unit an SM, and one more
    m = B.Matrix(R, K, R + K, eb=-21) if p == 4 else B.Matrix3(R, K, R + K, eb=-21)
    w = kernels.SeedWeight.from_matrices([m]) if p == 4 else kernels.SeedWeight3([m])
    x = B.bfr(np.random.default_rng(T).standard_normal((T, K)).astype(np.float32))
    assert np.array_equal(kernels.kt_mm(w, x, T, packed=False), kernels.kt_mm(w, x, T, packed=True))
