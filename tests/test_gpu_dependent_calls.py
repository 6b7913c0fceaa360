"""Calls that are dependent launches by themselves (router, gathers, combine, LM head and arg-max, prompt GEMM): queued one behind the other, with the
buffers of the previous round still in flight and kernels of another library in between, they give the bits of calls that are waited for one by one."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def ptr(t):
    return C.c_void_p(t.data_ptr() if t is not None else 0)


@pytest.mark.parametrize("p", [4, 3])
@pytest.mark.parametrize("T", [1, 8])
def test_a_layer_by_its_own_calls(p, T):
    import torch
    from nanoseedlm_b200 import kernels, lib as L
    from oracle import binding as B
    lib, G = L.load(), kernels.stream_table()
    d, ff, E, k = 512, 256, 12, 4
    if p == 4:
        stack = lambda R, K, s: kernels.SeedWeight.from_matrices([B.Matrix(R, K, s + e, eb=-20) for e in range(E)])
    else:
        stack = lambda R, K, s: kernels.SeedWeight3([B.Matrix3(R, K, s + e, eb=-20) for e in range(E)])
    gate, up, down = stack(ff, d, 1), stack(ff, d, 50), stack(d, ff, 99)
    fmt = L.MF_SEED4P4 if p == 4 else L.MF_SEED4
    gen = torch.Generator(device="cuda").manual_seed(3)
    xs = [torch.randn(T, d, generator=gen, device="cuda").to(torch.bfloat16).float() for _ in range(6)]
    ls = [torch.randn(T, E, generator=gen, device="cuda") for _ in range(6)]
    s = torch.cuda.Stream()
    x, logits, out = torch.zeros(T, d, device="cuda"), torch.zeros(T, E, device="cuda"), torch.zeros(T, d, device="cuda")
    ind, wt = torch.zeros(T, k, dtype=torch.int32, device="cuda"), torch.zeros(T, k, device="cuda")
    A, D = torch.zeros(T * k, ff, device="cuda"), torch.zeros(T * k, d, device="cuda")

    def run(wait):
        res = []
        torch.cuda.synchronize()
        with torch.cuda.stream(s):
            st = C.c_void_p(s.cuda_stream)
            done = (lambda: s.synchronize()) if wait else (lambda: None)
            for rep in range(4):
                for xi, li in zip(xs, ls):
                    x.mul_(0.0).add_(xi)               # another library's kernels before and after
                    logits.copy_(li)
                    done(); lib.nsl_route(st, E, k, ptr(logits), E, ptr(ind), ptr(wt), T)
                    done(); lib.kc_mv_gu(st, fmt, ptr(gate.table), ptr(up.table), d, ff, ptr(x), d, ptr(A), ff, ptr(ind), T * k, k, ptr(G))
                    done(); lib.kc_mv_sel(st, fmt, ptr(down.table), ff, d, ptr(A), ff, ptr(D), d, ptr(ind), T * k, 1, ptr(G))
                    done(); lib.kq4_moe_combine(st, d, k, ptr(D), ptr(wt), None, None, 0, ptr(out), T)
                    done(); res.append(out.clone())
        torch.cuda.synchronize()
        L.check()
        return torch.stack(res)

    assert torch.equal(run(False), run(True))


def test_prompt_product_head_and_tokens():
    import torch
    from nanoseedlm_b200 import kernels, lib as L, moe
    lib, G = L.load(), kernels.stream_table()
    K, V, T = 512, 9000, 8
    gen = torch.Generator(device="cuda").manual_seed(5)
    st = moe.ExpertStack.random_on_device(1, K, K, gen)
    w = L.WSlice()
    w.p[0], w.p[1], w.p[3], w.eb = st.seeds.data_ptr(), st.coefs.data_ptr(), st.codes.data_ptr(), -22
    codes = torch.randint(-2 ** 31, 2 ** 31 - 1, (V, K // 8), generator=gen, device="cuda", dtype=torch.int32)
    sc = (torch.rand((V, K // 64), generator=gen, device="cuda") * 0.02 + 0.001).to(torch.bfloat16)
    bi = (torch.rand((V, K // 64), generator=gen, device="cuda") * -0.2).to(torch.bfloat16)
    q = L.WSlice()
    q.p[0], q.p[1], q.p[2] = codes.data_ptr(), sc.data_ptr(), bi.data_ptr()
    xs = [torch.randn(n, K, generator=gen, device="cuda").to(torch.bfloat16).float() for n in (100, 9, 300, 40)]
    y, lg, tok = torch.zeros(300, K, device="cuda"), torch.zeros(T, V, device="cuda"), torch.zeros(T, dtype=torch.int32, device="cuda")

    def run(wait):
        res = []
        torch.cuda.synchronize()
        done = torch.cuda.synchronize if wait else (lambda: None)
        for rep in range(5):
            for x in xs:
                done(); lib.kc_mm(None, L.MF_SEED4P4, w, K, K, ptr(x), K, ptr(y), K, x.shape[0], 0, ptr(G))
                done(); lib.kc_mv(None, L.MF_Q4, q, K, V, ptr(y), K, ptr(lg), V, T, 0, None)
                done(); lib.kc_argmax(None, ptr(lg), ptr(tok), V, T)
                done(); res += [y[:x.shape[0]].clone().flatten(), lg.clone().flatten(), tok.float()]
        torch.cuda.synchronize()
        L.check()
        return torch.cat(res)

    assert torch.equal(run(False), run(True))


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
