"""Single-layer kernels of narrow layers (motifcl_b200/csrc/layer_kernels.cu) at the edges of their tiles: rows around 128,
columns around the tile widths, in_features that are no multiple of 16 or 64, token counts below one slice per CTA."""
import numpy as np
import pytest
import torch

from motifcl_b200 import synth

pytestmark = pytest.mark.gpu
SHAPES = [(16, 64, 32), (33, 68, 37), (127, 288, 288), (257, 108, 130), (300, 512, 96), (129, 1024, 200), (1000, 1020, 129), (2050, 80, 1536)]


@pytest.fixture(scope="module")
def ctx():
    from motifcl_b200 import Context
    c = Context.on_torch_stream(0)
    c.set_gemm_mode("tensor")
    yield c
    c.close()


def _layer(N, I, O, seed):
    rng = np.random.default_rng(seed)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    return (dev(synth.counters(77, seed, O, I).reshape(-1)), dev(rng.uniform(0.02, 0.2, O).astype(np.float32)),
            dev(rng.uniform(1e-4, 1e-2, O).astype(np.float32)), dev(rng.standard_normal((N, I)).astype(np.float32)),
            dev((rng.standard_normal((N, O)) * 0.02).astype(np.float32)))


# the last four: K cut over clusters of 8, 4 and 2, in parts that are not of one length, beside whole K
@pytest.mark.parametrize("N,I,O", SHAPES + [(40, 1024, 1025), (130, 100, 2047), (4096, 288, 1536), (600, 640, 301)])
def test_row_products_against_float64(ctx, N, I, O):
    st, sc, _, x, dy = _layer(N, I, O, N + I + O)
    w = torch.empty(O, I, device="cuda")
    ctx.counter_decode_weight(st, torch.ones_like(sc), w, I, O, 11)
    y, dx = torch.full((N, O), 7.0, device="cuda"), torch.full((N, I), 7.0, device="cuda")
    ctx.counter_forward(x, st, sc, y, N, I, O, 11)
    ctx.counter_backward_input(st, sc, dy, dx, N, I, O, 11)
    ctx.finish()
    ry = (x.double() @ w.double().T) * sc.double()
    rdx = (dy * sc).double() @ w.double()
    assert float((y - ry).norm() / ry.norm()) < 1e-6
    assert float((dx - rdx).norm() / rdx.norm()) < 1e-6


# cut over clusters of 8, 8 and 4 in one product at least, and whole K
@pytest.mark.parametrize("N,I,O", [(40, 1024, 1025), (130, 100, 2047), (600, 640, 301), (127, 288, 288)])
def test_row_sums_that_leave_fp32_are_infinities(ctx, N, I, O):
    """Row m of x has the signs of the digits of output m, row m of dy those of input m: every term of one sum is positive."""
    st, sc, _, x, dy = _layer(N, I, O, N + I + O)
    w = torch.empty(O, I, device="cuda")
    ctx.counter_decode_weight(st, torch.ones_like(sc), w, I, O, 11)
    ctx.finish()
    n, k = min(N, O), min(N, I)
    x[:n], dy[:k] = 1e37 * w[:n], 1e38 * w[:, :k].T              # no term leaves fp32 by itself
    y, dx = torch.full((N, O), 7.0, device="cuda"), torch.full((N, I), 7.0, device="cuda")
    torch.cuda.synchronize()
    ctx.counter_forward(x, st, sc, y, N, I, O, 11)
    ctx.counter_backward_input(st, sc, dy, dx, N, I, O, 11)
    ctx.finish()
    many = w.double().square().sum(dim=1)[:n] * 1e37 > 5e38
    assert bool(many.any()) and bool((y.diagonal()[:n][many] == float("inf")).all())
    far = (sc.double() @ w.double().square())[:k] * 1e38 > 1e39
    assert bool(far.any()) and bool((dx.diagonal()[:k][far] == float("inf")).all())


@pytest.mark.parametrize("lr_scale", [0.0, 1e-3])
@pytest.mark.parametrize("N,I,O", SHAPES)
def test_update_against_the_exact_path(ctx, N, I, O, lr_scale):
    res = []
    for mode in ("tensor", "exact"):
        st, sc, v, x, dy = _layer(N, I, O, N + I + O)
        p2 = torch.zeros(O, I // 16, dtype=torch.int32, device="cuda") if I % 16 == 0 else None
        ctx.set_gemm_mode(mode)
        try:
            ctx.counter_update_fused(st, sc, v, dy, x, p2, 11, I, O, N, 3e-3, lr_scale, 0.9, 1e-3, 99)
            ctx.finish()
        finally:
            ctx.set_gemm_mode("tensor")
        if p2 is not None:
            want = torch.empty_like(p2)
            ctx.counter_pack2(st, want, I, O, 11)
            ctx.finish()
            assert torch.equal(p2, want)
        res.append((st, sc, v))
    (st, sc, v), (est, esc, ev) = res
    assert float((st != est).double().mean()) <= 2e-4          # a rounding that falls the other way for a last-bit gradient difference
    assert float((sc - esc).norm() / esc.norm()) < 1e-6 and float((v - ev).norm() / ev.norm()) < 1e-5


@pytest.mark.parametrize("N", [32768, 32800, 98304, 300000, 500000])
def test_update_of_many_tokens(ctx, N):
    """dW of a long sum that grows all the way: an accumulator truncates less than a last bit for each of the 256 instructions that add
    leading products into it, and v (with rms_beta = 0 the mean square of a row of dW) shows twice that."""
    I, O = 64, 40
    g = torch.Generator(device="cuda").manual_seed(N)
    x, dy = torch.rand(N, I, device="cuda", generator=g) + 0.5, torch.rand(N, O, device="cuda", generator=g) * 0.02 + 0.01
    st, sc, v = torch.zeros(O * I // 4 * 3, dtype=torch.uint8, device="cuda"), torch.full((O,), 0.05, device="cuda"), torch.zeros(O, device="cuda")
    ctx.counter_update_fused(st, sc, v, dy, x, None, 11, I, O, N, 3e-3, 0.0, 0.0, 1e-3, 99)
    ctx.finish()
    want = (dy.double().T @ x.double()).square().mean(dim=1)
    assert float(((v.double() - want) / want).abs().max()) <= 2 * 256 * 2.0 ** -23


@pytest.mark.parametrize("N,I,O", [(40000, 288, 768), (40000, 768, 288), (8200, 1024, 1024), (5001, 1024, 1540), (70000, 288, 288), (33001, 512, 516)])
def test_both_routes_of_a_layer(N, I, O):
    """Token counts beyond those that the one-launch kernels take by themselves: split terms, or, where a recording keeps the workspace from
    growing, the one-launch kernels all the same; both against float64."""
    from motifcl_b200 import Context
    st, sc, v, x, dy = _layer(N, I, O, N + I)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        ctx = Context.on_torch_stream(0)
        w = torch.empty(O, I, device="cuda")
        ctx.counter_decode_weight(st, torch.ones_like(sc), w, I, O, 11)
        ctx.finish()
        wy, wdx = (x.double() @ w.double().T) * sc.double(), (dy * sc).double() @ w.double()
        wv = (dy.double().T @ x.double()).square().mean(dim=1)
        for recorded in (True, False):
            y, dx = torch.full((N, O), 7.0, device="cuda"), torch.full((N, I), 7.0, device="cuda")
            s2, c2, v2 = st.clone(), sc.clone(), v.clone()
            torch.cuda.synchronize()
            if recorded:
                ctx.batch_begin()
            ctx.counter_forward(x, st, sc, y, N, I, O, 11)
            ctx.counter_backward_input(st, sc, dy, dx, N, I, O, 11)
            ctx.counter_update_fused(s2, c2, v2, dy, x, None, 11, I, O, N, 3e-3, 0.0, 0.0, 1e-3, 99)
            if recorded:
                batch = ctx.batch_end()
                batch.launch()
            ctx.finish()
            if recorded:
                assert ctx.workspace_bytes == 0
                batch.close()
            assert float((y - wy).norm() / wy.norm()) < 1e-6 and float((dx - wdx).norm() / wdx.norm()) < 1e-6
            assert float(((v2.double() - wv) / wv).abs().max()) <= 2 * 256 * 2.0 ** -23
        ctx.close()


def test_layer_calls_under_a_capture_of_the_caller():
    """A graph that the caller captures on the context's stream: layer calls that would rather have workspace run without, and a call that
    cannot is refused without breaking the capture."""
    from motifcl_b200 import Context, MotifclCudaError
    N, I, O = 8200, 1024, 1024
    st, sc, v, x, dy = _layer(N, I, O, 4)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        ctx = Context.on_torch_stream(0)
        w, y, dx = torch.empty(O, I, device="cuda"), torch.empty(N, O, device="cuda"), torch.empty(N, I, device="cuda")
        ctx.counter_decode_weight(st, torch.ones_like(sc), w, I, O, 11)
        wy, wdx = (x.double() @ w.double().T) * sc.double(), (dy * sc).double() @ w.double()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        graph.capture_begin()
        try:
            ctx.counter_forward(x, st, sc, y, N, I, O, 11)
            ctx.counter_backward_input(st, sc, dy, dx, N, I, O, 11)
            with pytest.raises(MotifclCudaError):
                ctx.matmul_f32(x, w, y, N, I, O, trans_b=True)
        finally:
            graph.capture_end()
        for _ in range(2):
            y.zero_(), dx.zero_()
            graph.replay()
            ctx.finish()
            assert float((y - wy).norm() / wy.norm()) < 1e-6 and float((dx - wdx).norm() / wdx.norm()) < 1e-6
        del graph
        ctx.close()


@pytest.mark.parametrize("recorded", [False, True])
def test_launches_that_overlap_give_the_bits_of_launches_apart(recorded):
    """Every launch reads what the one before it wrote (a memset and a fork among them), many times over in buffers that are taken again."""
    from motifcl_b200 import Context
    stream = torch.cuda.Stream(device=0)
    with torch.cuda.stream(stream):
        ctx, lane = Context.on_torch_stream(0), Context(0)
        g = torch.Generator(device="cuda").manual_seed(5)
        N, D, F = 192, 288, 320
        x0 = torch.randn(N, D, device="cuda", generator=g)
        st0 = torch.randint(0, 256, (F * D // 4 * 3,), device="cuda", generator=g, dtype=torch.int32).to(torch.uint8)
        packed = torch.randn(N, 2 * F, device="cuda", generator=g)

        def state():
            s = {"x": x0.clone(), "st": st0.clone(), "scale": torch.full((F,), 0.07, device="cuda"), "v": torch.full((F,), 0.01, device="cuda")}
            for n, shape in (("h", (N, D)), ("r", (N, D)), ("y", (N, F)), ("dx", (N, D)), ("act", (N, F)), ("inv", (N,)), ("dw", (D,))):
                s[n] = torch.zeros(shape, device="cuda")
            return s

        def calls(s, apart):
            def after():
                if apart:
                    ctx.finish()
            one = s["scale"][:D]
            for _ in range(3):
                ctx.rmsnorm(s["x"], one, s["h"], N, D, 1e-5); after()
                ctx.rope(s["h"], s["r"], 2, N // 2, D, 6, 48); after()
                ctx.counter_forward(s["r"], s["st"], s["scale"], s["y"], N, D, F, 11); after()
                ctx.counter_backward_input(s["st"], s["scale"], s["y"], s["dx"], N, D, F, 11); after()
                ctx.counter_update_fused(s["st"], s["scale"], s["v"], s["y"], s["r"], None, 11, D, F, N, 3e-3, 0.05, 0.9, 1e-3, 77); after()
                ctx.swiglu(packed, s["act"], N, F); after()
                ctx.rmsnorm_backward_weight(s["dx"], s["r"], s["inv"], s["dw"], N, D, 1e-5); after()
                ctx.lane_fork(lane); ctx.lane_join(lane); after()
                ctx.rmsnorm_backward_x(s["dx"], one, s["r"], s["x"], N, D, 1e-5); after()
        a, b = state(), state()
        calls(a, True)
        ctx.finish()
        if recorded:
            ctx.batch_begin()
            calls(b, False)
            batch = ctx.batch_end()
            batch.launch()
            ctx.finish()
            batch.close()
        else:
            calls(b, False)
            ctx.finish()
        lane.close()
    for n in a:
        if n != "dw":                    # added up with atomics
            assert torch.equal(a[n], b[n]), n
    assert torch.isfinite(a["x"]).all() and not torch.equal(a["st"], st0)


@pytest.mark.parametrize("lr_scale", [0.0, 0.05])
@pytest.mark.parametrize("N,I,O", [(1, 16, 1), (33, 64, 32), (35, 68, 37), (17, 1000, 149), (8, 1024, 300), (129, 128, 200), (1000, 64, 64), (65, 48, 1300), (7, 4, 2)])
def test_small_products_and_updates_in_the_order_of_the_reference(orc, N, I, O, lr_scale):
    """Below 2^22 multiply-adds, bit for bit: tokens and features ascending, multiply and add rounded apart, whatever part of a tile of
    16, a slice of 64 or a set of eight tokens exists; the update in one launch, with and without 2-bit words."""
    from motifcl_b200 import Context
    st, sc, v, x, dy = _layer(N, I, O, N + I + O)
    hy = (3e-3, lr_scale, 0.9, 1e-3, 4242)
    own = Context.on_torch_stream(0)
    y, dx = torch.full((N, O), 7.0, device="cuda"), torch.full((N, I), 7.0, device="cuda")
    p2 = torch.zeros(O, I // 16, dtype=torch.int32, device="cuda") if I % 16 == 0 else None
    h = lambda a: a.cpu().numpy().copy()
    hst, hsc, hv, hx, hdy = h(st), h(sc), h(v), h(x), h(dy)
    own.counter_forward(x, st, sc, y, N, I, O, 11)
    own.counter_backward_input(st, sc, dy, dx, N, I, O, 11)
    before = own.launch_count
    own.counter_update_fused(st, sc, v, dy, x, p2, 11, I, O, N, *hy)
    own.finish()
    assert own.launch_count - before == 1
    assert np.array_equal(h(y).view(np.uint32), orc.forward(hx, hst, hsc, 11, O).view(np.uint32))
    assert np.array_equal(h(dx).view(np.uint32), orc.backward_input(hdy, hst, hsc, 11, I).view(np.uint32))
    e = orc.update_fused(hst, hsc, hv, hdy, hx, 11, *hy)
    assert np.array_equal(h(st), e[0])
    assert np.array_equal(h(sc).view(np.uint32), e[1].view(np.uint32)) and np.array_equal(h(v).view(np.uint32), e[2].view(np.uint32))
    if p2 is not None:
        assert np.array_equal(h(p2).view(np.uint32).reshape(-1), np.asarray(e[3]).reshape(-1))
    own.close()
