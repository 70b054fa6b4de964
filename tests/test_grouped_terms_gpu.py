"""Weight gradients of layers stepped together whose operands exceed L2: all terms of a k-tile from one slot."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("I,O,tokens,layers", [(288, 288, 32769, 3), (768, 288, 20000, 3), (64, 1000, 24001, 3), (320, 132, 60000, 3)])
def test_grad_w_of_a_large_group(I, O, tokens, layers):
    from motifcl_b200 import Context
    from motifcl_b200.runtime import linear_descs
    stream = torch.cuda.Stream(device=0)
    with torch.cuda.stream(stream):
        ctx = Context.on_torch_stream(0)
        g = torch.Generator(device=DEV).manual_seed(I + O)
        ls = []
        for _ in range(layers):
            ls.append(dict(x=torch.randn(tokens, I, device=DEV, generator=g), grad_out=torch.randn(tokens, O, device=DEV, generator=g) * 0.02,
                           state=torch.randint(0, 256, (O * I // 4 * 3,), device=DEV, generator=g, dtype=torch.int32).to(torch.uint8),
                           scale=torch.full((O,), 0.05, device=DEV), v=torch.zeros(O, device=DEV), y=torch.empty(tokens, O, device=DEV),
                           grad_x=torch.empty(tokens, I, device=DEV), grad_w=torch.full((O, I), 7.0, device=DEV), packed2_out=None))
        descs = linear_descs([dict(l, in_features=I, out_features=O, batch=tokens, update_rows=0) for l in ls])
        ctx.counter_linear_step_many(descs, 11, 3e-3, 0.0, 0.9, 1e-3, 1)
        for l in ls:
            want = l["grad_out"].double().T @ l["x"].double()
            assert float((l["grad_w"].double() - want).norm() / want.norm()) <= 5e-6
            assert float((l["grad_w"].double() - want).abs().max() / want.square().mean().sqrt()) <= 5e-5


def test_contractions_side_by_side_and_again():
    """Two contexts' contractions at once, so that CTAs start late and find their items taken, then again: the counters are back at
    zero.  An item's result does not depend on who computes it: all runs equal the first, bit for bit."""
    from motifcl_b200 import Context
    from motifcl_b200.runtime import linear_descs
    sides = []
    for I, O, tokens, layers in ((288, 768, 8192, 6), (2048, 1024, 3000, 2), (512, 512, 777, 9)):
        stream = torch.cuda.Stream(device=0)
        with torch.cuda.stream(stream):
            ctx = Context.on_torch_stream(0)
            g = torch.Generator(device=DEV).manual_seed(I)
            ls = [dict(x=torch.randn(tokens, I, device=DEV, generator=g), grad_out=torch.randn(tokens, O, device=DEV, generator=g),
                       state=torch.randint(0, 256, (O * I // 4 * 3,), device=DEV, generator=g, dtype=torch.int32).to(torch.uint8),
                       scale=torch.full((O,), 0.05, device=DEV), v=torch.zeros(O, device=DEV), y=torch.empty(tokens, O, device=DEV),
                       grad_x=torch.empty(tokens, I, device=DEV), grad_w=torch.empty(O, I, device=DEV), packed2_out=None) for _ in range(layers)]
            descs = linear_descs([dict(l, in_features=I, out_features=O, batch=tokens, update_rows=0) for l in ls])
            ctx.counter_linear_step_many(descs, 11, 3e-3, 0.0, 0.9, 1e-3, 1)
            ctx.finish()
            w = torch.empty(O, I, device=DEV)
            ctx.counter_decode_weight(ls[-1]["state"], ls[-1]["scale"], w, I, O, 11)
            ctx.finish()
            want = ls[-1]["x"].double() @ w.double().T
            assert float((ls[-1]["y"].double() - want).norm() / want.norm()) <= 1e-6
            sides.append((ctx, descs, ls, [{n: l[n].clone() for n in ("y", "grad_x", "grad_w")} for l in ls], stream))
    torch.cuda.synchronize()
    for _ in range(5):
        for ctx, descs, ls, first, stream in sides:
            with torch.cuda.stream(stream):
                for l in ls:
                    l["y"].fill_(7.0), l["grad_x"].fill_(7.0), l["grad_w"].fill_(7.0)
                ctx.counter_linear_step_many(descs, 11, 3e-3, 0.0, 0.9, 1e-3, 1)
        for ctx, _, ls, first, _ in sides:
            ctx.finish()
            for l, f in zip(ls, first):
                assert all(torch.equal(l[n], f[n]) for n in f)


@pytest.mark.parametrize("N,I,O", [(40, 1088, 1156), (70, 4096, 1028), (300, 2048, 1100), (777, 1024, 3076), (161, 1156, 4100), (1030, 1536, 1032)])
def test_row_products_on_tokens_that_leave_a_tile_ragged(N, I, O):
    """Tokens as columns of the product (digits times activations) or as its rows, whichever wastes less: rows 2^-80 to 2^80 of one another
    keep their bits (24 of the row's largest element, by as many as are added up), an infinity stays in its row."""
    from motifcl_b200 import Context
    rng = np.random.default_rng(N + I + O)
    ctx = Context.on_torch_stream(0)
    ctx.set_gemm_mode("tensor")
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    st, sc = dev(rng.integers(0, 256, O * I // 4 * 3, dtype=np.uint8)), dev(rng.uniform(0.02, 0.2, O).astype(np.float32))
    w = torch.empty(O, I, device="cuda")
    ctx.counter_decode_weight(st, torch.ones_like(sc), w, I, O, 11)
    rows = np.exp2(rng.integers(-80, 81, (N, 1))).astype(np.float32)
    x, dy = dev(rng.standard_normal((N, I)).astype(np.float32) * rows), dev(rng.standard_normal((N, O)).astype(np.float32) * rows)
    x[N // 2, 3] = float("inf")
    y, dx = torch.full((N, O), 7.0, device="cuda"), torch.full((N, I), 7.0, device="cuda")
    ctx.counter_forward(x, st, sc, y, N, I, O, 11)
    ctx.counter_backward_input(st, sc, dy, dx, N, I, O, 11)
    ctx.finish()
    keep = torch.arange(N, device="cuda") != N // 2
    for got, want in ((y, (x.double() @ w.double().T) * sc.double()), (dx, (dy * sc).double() @ w.double())):
        err = (got[keep].double() - want[keep]).norm(dim=1) / want[keep].norm(dim=1)
        assert float(err.max()) < 1e-6
    assert not torch.isfinite(y[N // 2]).all() and torch.isfinite(y[keep]).all()
    ctx.close()
