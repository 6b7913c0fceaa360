"""Calls that are dependent launches by themselves (router, gathers, combine, LM head and arg-max, prompt GEMM): queued one behind the other or captured in a
graph, with the buffers of the previous round still in flight, they give the bits of calls that are waited for one by one; and the switch that decides."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def ptr(t):
    return C.c_void_p(t.data_ptr() if t is not None else 0)


def three_ways(calls, results):
    """calls(stream, done) issues a whole sequence, done() after each call; results() gives its outputs.  -> the outputs where each call is waited for;
    where the sequence is queued before its first call starts (large products run in front of it meanwhile); and of a captured graph, replayed twice."""
    import torch
    got, s = [], torch.cuda.Stream()
    st = C.c_void_p(s.cuda_stream)
    a = torch.randn(8192, 8192, device="cuda").to(torch.bfloat16)
    b = torch.empty_like(a)
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        for r in results(): r.zero_()
        calls(st, s.synchronize)
        s.synchronize()
        got.append([r.clone() for r in results()])
        for attempt in range(4):      # (again where the host was held up meanwhile)
            for r in results(): r.zero_()
            for _ in range(12): torch.mm(a, a, out=b)
            begin = torch.cuda.Event()
            begin.record(s)
            calls(st, lambda: None)
            queued = not begin.query()      # nothing of the sequence has started yet
            s.synchronize()
            if queued: break
        assert queued
        got.append([r.clone() for r in results()])
    rt, graph, exe = C.CDLL("libcudart.so.12"), C.c_void_p(), C.c_void_p()
    assert rt.cudaStreamBeginCapture(st, 2) == 0
    calls(st, lambda: None)
    assert rt.cudaStreamEndCapture(st, C.byref(graph)) == 0 and rt.cudaGraphInstantiate(C.byref(exe), graph, C.c_ulonglong(0)) == 0
    with torch.cuda.stream(s):
        for r in results(): r.zero_()
        for _ in range(2): assert rt.cudaGraphLaunch(exe, st) == 0
        s.synchronize()
        got.append([r.clone() for r in results()])
    rt.cudaGraphExecDestroy(exe)
    rt.cudaGraphDestroy(graph)
    return got


@pytest.mark.parametrize("p", [4, 3])
@pytest.mark.parametrize("T,d,ff,E,k", [(1, 512, 256, 12, 4), (8, 512, 256, 12, 4), (8, 1536, 704, 60, 4), (3, 520, 264, 12, 4), (32, 1024, 512, 16, 4)])
def test_a_layer_by_its_own_calls(p, T, d, ff, E, k):
    """Rounds of router, gate + up, down and combine over the same buffers, with nothing in between: a round overwrites what the round before has just read."""
    import torch
    from nanoseedlm_b200 import kernels, lib as L
    from oracle import binding as B
    lib, G = L.load(), kernels.stream_table()
    if p == 4:
        stack = lambda R, K, s: kernels.SeedWeight.from_matrices([B.Matrix(R, K, s + e, eb=-20) for e in range(E)])
    else:
        stack = lambda R, K, s: kernels.SeedWeight3([B.Matrix3(R, K, s + e, eb=-20) for e in range(E)])
    gate, up, down = stack(ff, d, 1), stack(ff, d, 50), stack(d, ff, 99)
    fmt = L.MF_SEED4P4 if p == 4 else L.MF_SEED4
    gen = torch.Generator(device="cuda").manual_seed(3)
    rounds = 12
    x = torch.randn(rounds, T, d, generator=gen, device="cuda").to(torch.bfloat16).float()
    logits, out = torch.randn(rounds, T, E, generator=gen, device="cuda"), torch.zeros(rounds, T, d, device="cuda")
    ind, wt = torch.zeros(T, k, dtype=torch.int32, device="cuda"), torch.zeros(T, k, device="cuda")
    A, D = torch.zeros(T * k, ff, device="cuda"), torch.zeros(T * k, d, device="cuda")

    def calls(st, done):
        for i in range(rounds):
            lib.nsl_route(st, E, k, ptr(logits[i]), E, ptr(ind), ptr(wt), T); done()
            lib.kc_mv_gu(st, fmt, ptr(gate.table), ptr(up.table), d, ff, ptr(x[i]), d, ptr(A), ff, ptr(ind), T * k, k, ptr(G)); done()
            lib.kc_mv_sel(st, fmt, ptr(down.table), ff, d, ptr(A), ff, ptr(D), d, ptr(ind), T * k, 1, ptr(G)); done()
            lib.kq4_moe_combine(st, d, k, ptr(D), ptr(wt), None, None, 0, ptr(out[i]), T); done()

    waited, queued, graph = three_ways(calls, lambda: [out, ind, wt, A, D])
    L.check()
    assert bool(waited[0].any())
    for a, b, c in zip(waited, queued, graph): assert torch.equal(a, b) and torch.equal(a, c)


# The head's forms: K split over the warps (two widths), streams through shared memory, streams from memory; the arg-max of a cluster a row and of a block a row.
@pytest.mark.parametrize("K,V", [(2048, 24064), (4096, 13000), (1536, 30000), (1216, 24064), (512, 9000)])
def test_prompt_product_head_and_tokens(K, V):
    import torch
    from nanoseedlm_b200 import kernels, lib as L, moe
    lib, G, T = L.load(), kernels.stream_table(), 8
    gen = torch.Generator(device="cuda").manual_seed(5)
    st4 = moe.ExpertStack.random_on_device(1, K, K, gen)
    w = L.WSlice()
    w.p[0], w.p[1], w.p[3], w.eb = st4.seeds.data_ptr(), st4.coefs.data_ptr(), st4.codes.data_ptr(), -22
    codes = torch.randint(-2 ** 31, 2 ** 31 - 1, (V, K // 8), generator=gen, device="cuda", dtype=torch.int32)
    sc = (torch.rand((V, K // 64), generator=gen, device="cuda") * 0.02 + 0.001).to(torch.bfloat16)
    bi = (torch.rand((V, K // 64), generator=gen, device="cuda") * -0.2).to(torch.bfloat16)
    q = L.WSlice()
    q.p[0], q.p[1], q.p[2] = codes.data_ptr(), sc.data_ptr(), bi.data_ptr()
    xs = [torch.randn(n, K, generator=gen, device="cuda").to(torch.bfloat16).float() for n in (100, 9, 300, 40, 65, 513)]
    y, lg = torch.zeros(513, K, device="cuda"), torch.zeros(T, V, device="cuda")
    tok, prob = torch.zeros(len(xs), T, dtype=torch.int32, device="cuda"), torch.zeros(len(xs), T, device="cuda")      # a probability depends on every logit

    def calls(st, done):
        for i, x in enumerate(xs):
            lib.kc_mm(st, L.MF_SEED4P4, w, K, K, ptr(x), K, ptr(y), K, x.shape[0], 0, ptr(G)); done()
            lib.kc_mv(st, L.MF_Q4, q, K, V, ptr(y), K, ptr(lg), V, T, 0, None); done()
            lib.kc_argmax_p(st, ptr(lg), ptr(tok[i]), ptr(prob[i]), V, T); done()

    waited, queued, graph = three_ways(calls, lambda: [tok, prob, y, lg])
    L.check()
    assert bool(waited[0].any()) and bool(torch.isfinite(waited[3]).all())
    for a, b, c in zip(waited, queued, graph): assert torch.equal(a, b) and torch.equal(a, c)


@pytest.fixture
def switch():
    """nsl_dependent_launch, set back afterwards."""
    from nanoseedlm_b200 import lib as L
    lib = L.load()
    before = lib.nsl_dependent_launch_state()
    yield lib.nsl_dependent_launch
    lib.nsl_dependent_launch(before)


def edges_of(calls):
    """The calls captured into a graph of one stream: (programmatic edges, other edges)."""
    import torch
    rt = C.CDLL("libcudart.so.12")
    s, graph = torch.cuda.Stream(), C.c_void_p()
    torch.cuda.synchronize()
    assert rt.cudaStreamBeginCapture(C.c_void_p(s.cuda_stream), 2) == 0
    calls(C.c_void_p(s.cuda_stream))
    assert rt.cudaStreamEndCapture(C.c_void_p(s.cuda_stream), C.byref(graph)) == 0
    n = C.c_size_t(0)
    assert rt.cudaGraphGetEdges_v2(graph, None, None, None, C.byref(n)) == 0
    f, t, data = (C.c_void_p * n.value)(), (C.c_void_p * n.value)(), (C.c_uint8 * (8 * n.value))()      # an edge's data: from, to, type, 5 bytes reserved
    assert rt.cudaGraphGetEdges_v2(graph, f, t, data, C.byref(n)) == 0
    rt.cudaGraphDestroy(graph)
    kinds = [data[8 * i + 2] for i in range(n.value)]
    return sum(k == 1 for k in kinds), sum(k != 1 for k in kinds)


class Layer:
    """A SEED4P4 layer by its own calls on device buffers."""

    def __init__(self, T, d=512, ff=256, E=12, k=4):
        import torch
        from nanoseedlm_b200 import kernels, lib as L, moe
        gen = torch.Generator(device="cuda").manual_seed(7)
        self.lib, self.G, self.d, self.ff, self.E, self.k, self.T = L.load(), kernels.stream_table(), d, ff, E, k, T
        self.gate, self.up, self.down = (moe.ExpertStack.random_on_device(E, r, c, gen) for r, c in ((ff, d), (ff, d), (d, ff)))
        self.x = torch.randn(T, d, generator=gen, device="cuda").to(torch.bfloat16).float()
        self.logits = torch.randn(T, E, generator=gen, device="cuda")
        self.ind, self.wt = torch.zeros(T, k, dtype=torch.int32, device="cuda"), torch.zeros(T, k, device="cuda")
        self.A, self.D, self.out = torch.zeros(T * k, ff, device="cuda"), torch.zeros(T * k, d, device="cuda"), torch.zeros(T, d, device="cuda")

    def calls(self, s, G=None):
        from nanoseedlm_b200 import lib as L
        G, f = ptr(self.G if G is None else G), L.MF_SEED4P4
        self.lib.nsl_route(s, self.E, self.k, ptr(self.logits), self.E, ptr(self.ind), ptr(self.wt), self.T)
        self.lib.kc_mv_gu(s, f, ptr(self.gate.table), ptr(self.up.table), self.d, self.ff, ptr(self.x), self.d, ptr(self.A), self.ff, ptr(self.ind), self.T * self.k,
                          self.k, G)
        self.lib.kc_mv_sel(s, f, ptr(self.down.table), self.ff, self.d, ptr(self.A), self.ff, ptr(self.D), self.d, ptr(self.ind), self.T * self.k, 1, G)
        self.lib.kq4_moe_combine(s, self.d, self.k, ptr(self.D), ptr(self.wt), None, None, 0, ptr(self.out), self.T)


def test_the_switch(switch):
    """0: ordinary launches; positive: dependent ones; negative, and at the start: each entry point's own choice.  The bits are the same."""
    import torch
    layer, res = Layer(3), []
    layer.calls(None)      # (functions are loaded before a capture)
    assert edges_of(layer.calls) == (3, 0)
    for on, edges in ((0, (0, 3)), (1, (3, 0)), (-1, (3, 0)), (0, (0, 3))):
        switch(on)
        assert layer.lib.nsl_dependent_launch_state() == on
        assert edges_of(layer.calls) == edges
        layer.out.zero_()
        layer.calls(C.c_void_p(torch.cuda.current_stream().cuda_stream))
        res.append(layer.out.clone())
    assert all(torch.equal(r, res[0]) for r in res) and bool(res[0].any())


@pytest.mark.parametrize("kind,K,R,T", [("pair", 512, 256, 4), ("items", 1536, 256, 4), ("grp", 512, 256, 64), ("generic", 520, 256, 2), ("mma", 512, 256, 9),
                                        ("gemm", 512, 256, 100), ("gemm", 520, 256, 100)])
def test_a_table_made_by_the_kernel_before(kind, K, R, T):
    """A call that is a dependent launch by its own choice may use a stream table that the kernel before it has made, one that lets its dependents
    go early included (kc_pack_input_bf16: the table's halves as bf16 values)."""
    import torch
    from nanoseedlm_b200 import lib as L, moe, kernels
    lib, E, k = L.load(), 6, 4
    G = kernels.stream_table()
    halves = (G.view(torch.int16).to(torch.int32) << 16).view(torch.float32)
    made, want = torch.zeros_like(G), torch.zeros_like(G)
    gen = torch.Generator(device="cuda").manual_seed(K + T)
    st = moe.ExpertStack.random_on_device(E, R, K, gen)
    x = torch.randn(T, K, generator=gen, device="cuda").to(torch.bfloat16).float()
    sel = torch.randint(0, E, (T * k,), generator=gen, device="cuda", dtype=torch.int32)
    busy = torch.randn(2048, 2048, device="cuda")
    rows = T if kind in ("mma", "gemm") else T * k
    w = L.WSlice()
    w.p[0], w.p[1], w.p[3], w.eb = st.seeds.data_ptr(), st.coefs.data_ptr(), st.codes.data_ptr(), -22
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)

    def calls(y, y2, table):
        if kind in ("mma", "gemm"):
            lib.kc_mm(s, L.MF_SEED4P4, w, K, R, ptr(x), K, ptr(y), R, T, 0, ptr(table))
            return
        lib.kc_mv_sel(s, L.MF_SEED4P4, ptr(st.table), K, R, ptr(x), K, ptr(y), R, ptr(sel), T * k, k, ptr(table))
        lib.kc_mv_gu(s, L.MF_SEED4P4, ptr(st.table), ptr(st.table), K, R, ptr(x), K, ptr(y2), R, ptr(sel), T * k, k, ptr(table))

    lib.kc_pack_input_bf16(s, ptr(halves), ptr(want), halves.numel())
    torch.cuda.synchronize()
    ref = [torch.zeros(rows, R, device="cuda") for _ in range(2)]
    calls(*ref, want)
    torch.cuda.synchronize()
    for _ in range(5):
        got = [torch.zeros(rows, R, device="cuda") for _ in range(2)]
        made.zero_()
        for _ in range(4): busy @ busy      # the host gets ahead, so that the calls are queued when the table is made
        lib.kc_pack_input_bf16(s, ptr(halves), ptr(made), halves.numel())
        calls(*got, made)
        torch.cuda.synchronize()
        assert torch.equal(got[0], ref[0]) and torch.equal(got[1], ref[1]) and bool(ref[0].any())
    L.check()


def bf16_product():
    import torch
    from nanoseedlm_b200 import lib as L
    lib, K, R, T = L.load(), 256, 384, 100      # (format 0: stored BF16)
    gen = torch.Generator(device="cuda").manual_seed(11)
    wb, x = torch.randn(R, K, generator=gen, device="cuda").to(torch.bfloat16), torch.randn(T, K, generator=gen, device="cuda").to(torch.bfloat16).float()
    y, w = torch.zeros(T, R, device="cuda"), L.WSlice()
    w.p[0] = wb.data_ptr()
    return lambda s, rows: lib.kc_mm(s, 0, w, K, R, ptr(x), K, ptr(y), R, rows, 0, None), (wb, x, y)


@pytest.mark.parametrize("rows", [100, 9])      # the tile GEMM, the decode batch's kernel
def test_products_of_stored_bf16_weights_are_ordinary_launches(switch, rows):
    import torch
    call, (wb, x, y) = bf16_product()

    def both(s):
        call(s, rows)
        call(s, rows)

    both(None)
    assert edges_of(both) == (0, 1)
    switch(1)
    assert edges_of(both) == (1, 0)
    switch(0)
    assert edges_of(both) == (0, 1)
    torch.cuda.synchronize()
    ref = x[:rows].double() @ wb.double().T      # f32 sums of 256 products (at most 256 x 2^-24 of their magnitudes' sum) and one rounding to bf16 (8 significant bits: 2^-8)
    assert bool(((y[:rows].double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1.01 * 2.0 ** -16 * (x[:rows].double().abs() @ wb.double().abs().T)).all())


def test_calls_behind_an_event(switch):
    """The layer on a second stream that waits for the first one's event, joined again behind it: queued, and as a fork and join in a graph."""
    import torch
    layer = Layer(3)
    src, x0 = layer.x.clone(), torch.zeros_like(layer.x)
    big = torch.randn(4096, 4096, device="cuda")
    layer.calls(None)
    torch.cuda.synchronize()
    want = layer.out.clone()
    assert bool(want.any())
    total = torch.zeros_like(want)
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()

    def fork_and_join():
        ev1, ev2 = torch.cuda.Event(), torch.cuda.Event()
        with torch.cuda.stream(s1):
            layer.x.zero_()
            layer.x.copy_(src)
            ev1.record(s1)
            s2.wait_event(ev1)
            layer.calls(C.c_void_p(s2.cuda_stream))
            ev2.record(s2)
            s1.wait_event(ev2)
            total.add_(layer.out)

    for on in (-1, 1, 0):
        switch(on)
        total.zero_()
        layer.out.zero_()
        torch.cuda.synchronize()
        with torch.cuda.stream(s1):
            for _ in range(4): torch.mm(big, big)
        for _ in range(4): fork_and_join()
        torch.cuda.synchronize()
        assert torch.equal(total, want * 4), on
        total.zero_()
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s1):
            for _ in range(2): fork_and_join()
        for _ in range(2): g.replay()
        torch.cuda.synchronize()
        assert torch.equal(total, want * 4), on


def test_the_switch_and_a_layer_handle_beside_it(switch):
    """Calls with the switch turned between them, beside a layer whose own launches are ordinary: the bits stay."""
    import torch
    from nanoseedlm_b200 import moe
    layer, gen = Layer(8), torch.Generator(device="cuda").manual_seed(1)
    m = moe.Moe(moe.DeviceLayer.random_on_device(512, 256, 12, gen), 4, 8)
    x, lg, out = torch.randn(8, 512, generator=gen, device="cuda"), torch.randn(8, 12, generator=gen, device="cuda"), torch.zeros(8, 512, device="cuda")
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    refs = []
    for pdl in (1, 0):
        m.lib.nsl_moe_set_dependent_launch(m.h, pdl)
        for on in (0, -1, 1, -1):
            switch(on)
            layer.out.zero_()
            out.zero_()
            for _ in range(3):
                layer.calls(s)
                m.forward_dev(x, lg, out)
                switch(on if _ else 0)
            assert layer.lib.nsl_dependent_launch_state() == on
            refs.append((layer.out.clone(), out.clone()))
    m.close()
    assert all(torch.equal(a, refs[0][0]) and torch.equal(b, refs[0][1]) for a, b in refs) and bool(refs[0][0].any()) and bool(refs[0][1].any())
