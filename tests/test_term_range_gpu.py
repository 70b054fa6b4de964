"""Products of fp32 tensors whose magnitudes are spread: an element far above the others, wherever it lies, and the gradients of
a classifier.  Every product is compared with float64.  The bound: 2^-22 for the terms of both operands, and for each tensor-core
instruction that adds into one accumulator half a last bit of what it holds, 2^-24, because it truncates and one large term
may fill it from the start (at most 64 k-tiles of 64, three products of four instructions each)."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from motifcl_b200 import Context
    c = Context.on_torch_stream(0)
    c.set_gemm_mode("tensor")
    yield c
    c.close()


def _bound(k):
    return 2.0 ** -22 + 2.0 ** -24 * 12 * min(64, (k + 63) // 64)


def _row_errors(c, want):
    return (c.double() - want).norm(dim=1) / want.norm(dim=1)


@pytest.mark.parametrize("shift", [7, 8, 9, 10, 20])
@pytest.mark.parametrize("row,col", [(0, 511), (517, 301), (1023, 0)])
def test_one_element_above_a_flat_tensor(ctx, shift, row, col):
    """Magnitudes in [1, 2) and one of (2 - 2^-23) 2^shift: it may lie outside anything that looks at a part of the tensor."""
    M, K, N = 1024, 512, 96
    g = torch.Generator(device="cuda").manual_seed(shift)
    a = (1.0 + torch.rand(M, K, device="cuda", generator=g) * 0.999) * torch.sign(torch.randn(M, K, device="cuda", generator=g))
    a[row, col] = (2.0 - 2.0 ** -23) * 2.0 ** shift
    b, bt = torch.randn(K, N, device="cuda", generator=g), torch.randn(M, N, device="cuda", generator=g)
    c, ct = torch.empty(M, N, device="cuda"), torch.empty(K, N, device="cuda")
    ctx.matmul_f32(a, b, c, M, K, N)                              # contraction along the rows of a
    ctx.matmul_f32(a, bt, ct, K, M, N, trans_a=True)              # and along its columns
    ctx.finish()
    assert float(_row_errors(c, a.double() @ b.double()).max()) <= _bound(K)
    assert float(_row_errors(ct, a.double().T @ bt.double()).max()) <= _bound(M)


@pytest.mark.parametrize("tokens", [4096, 2048, 777])
def test_classifier_gradients(ctx, tokens):
    """The largest elements of a cross-entropy gradient are those of the targets, one in a row of 32000."""
    D, V = 288, 32000
    for seed in range(10):
        g = torch.Generator(device="cuda").manual_seed(seed)
        h, w = torch.randn(tokens, D, device="cuda", generator=g), torch.randn(V, D, device="cuda", generator=g) * D ** -0.5
        targets = torch.randint(0, V, (tokens,), device="cuda", generator=g, dtype=torch.int32)
        logits, grad, dh, dw = torch.empty(tokens, V, device="cuda"), torch.empty(tokens, V, device="cuda"), torch.empty_like(h), torch.empty_like(w)
        ctx.matmul_f32(h, w, logits, tokens, D, V, trans_b=True)
        ctx.softmax_cross_entropy_backward(logits, targets, torch.ones(1, device="cuda"), grad, tokens, V)
        ctx.matmul_f32(grad, w, dh, tokens, V, D)
        ctx.matmul_f32(grad, h, dw, V, tokens, D, trans_a=True)
        ctx.finish()
        for got, want, k in ((logits, h.double() @ w.double().T, D), (dh, grad.double() @ w.double(), V), (dw, grad.double().T @ h.double(), tokens)):
            assert float((got.double() - want).norm() / want.norm()) <= _bound(k)


def _linear(tokens, I, O, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    state = torch.randint(0, 256, (O * I // 4 * 3,), device="cuda", generator=g, dtype=torch.int32).to(torch.uint8)
    scale = torch.rand(O, device="cuda", generator=g) * 0.1 + 0.02
    return state, scale, torch.randn(tokens, I, device="cuda", generator=g), torch.randn(tokens, O, device="cuda", generator=g) * 0.02


def _products(ctx, state, scale, x, dy, grouped):
    """Y, dX and dW of one layer by its own call (grouped = 0) or of several at once."""
    from motifcl_b200.runtime import linear_descs
    (N, I), O = x.shape, dy.shape[1]
    y, dx, dw = torch.full((N, O), 7.0, device="cuda"), torch.full((N, I), 7.0, device="cuda"), torch.full((O, I), 7.0, device="cuda")
    one = dict(x=x, grad_out=dy, state=state, scale=scale, v=torch.zeros(O, device="cuda"), y=y, grad_x=dx, grad_w=dw, packed2_out=None,
               in_features=I, out_features=O, batch=N, update_rows=0)
    more = [dict(one, y=torch.empty_like(y), grad_x=torch.empty_like(dx), grad_w=torch.empty_like(dw)) for _ in range(grouped)]
    ctx.counter_linear_step_many(linear_descs([one] + more), 11, 3e-3, 0.0, 0.9, 1e-3, 1)
    w = torch.empty(O, I, device="cuda")
    ctx.counter_decode_weight(state, torch.ones_like(scale), w, I, O, 11)
    ctx.finish()
    return y, dx, dw, (x.double() @ w.double().T) * scale.double(), (dy * scale).double() @ w.double(), dy.double().T @ x.double()


@pytest.mark.parametrize("grouped", [0, 2])
@pytest.mark.parametrize("down", [20, 28, 36, 60, 100])
@pytest.mark.parametrize("tokens,I,O", [(300, 288, 96), (515, 1028, 2052), (130, 64, 8200)])
def test_rows_far_below_the_largest(ctx, tokens, I, O, down, grouped):
    """Each row of Y and dX has the relative error of a tensor of its own, whatever the other rows are."""
    state, scale, x, dy = _linear(tokens, I, O, down)
    small = torch.zeros(tokens, 1, device="cuda", dtype=torch.bool)
    small[1::3] = True
    x, dy = torch.where(small, x * 2.0 ** -down, x), torch.where(small.flip(0), dy * 2.0 ** -down, dy)
    y, dx, dw, wy, wdx, wdw = _products(ctx, state, scale, x, dy, grouped)
    assert float(_row_errors(y, wy).max()) <= 1e-6                # digits are exact; truncation of 2.7e-9 for each of 4 K / 64 instructions
    assert float(_row_errors(dx, wdx).max()) <= 4e-6
    assert float((dw.double() - wdw).norm() / wdw.norm()) <= _bound(tokens)


@pytest.mark.parametrize("grouped", [0, 2])
@pytest.mark.parametrize("tokens,I,O", [(300, 288, 96), (515, 1028, 2052), (130, 64, 8200)])
@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan"), 1e30, 3e38])
def test_one_bad_element_stays_in_its_row(ctx, tokens, I, O, value, grouped):
    state, scale, x, dy = _linear(tokens, I, O, 3)
    row, col = 77, 5
    for tensor in (x, dy):
        saved = float(tensor[row, col])
        tensor[row, col] = value
        y, dx, dw, wy, wdx, wdw = _products(ctx, state, scale, x, dy, grouped)
        tensor[row, col] = saved
        others = torch.arange(tokens, device="cuda") != row
        assert float(_row_errors(y, wy)[others].max()) <= 1e-6
        assert float(_row_errors(dx, wdx)[others].max()) <= 4e-6
        if not math.isfinite(value):                              # the element's column of dW, and no other
            rest = torch.ones_like(dw, dtype=torch.bool)
            if tensor is x:
                rest[:, col] = False
            else:
                rest[col, :] = False
            assert not torch.isfinite(dw[~rest]).any()
            e = (dw.double() - wdw)[rest]
            assert float(e.norm() / wdw[rest].norm()) <= _bound(tokens)


def test_products_at_the_ends_of_fp32(ctx):
    """Operands near the largest and the smallest normal values whose products are ordinary numbers, in every orientation."""
    M, K, N = 200, 520, 136
    g = torch.Generator(device="cuda").manual_seed(1)
    for up in (100, 120, -100, -120):
        a, b = torch.randn(M, K, device="cuda", generator=g) * 2.0 ** up, torch.randn(K, N, device="cuda", generator=g) * 2.0 ** -up
        want = a.double() @ b.double()
        for ta, tb in ((0, 0), (1, 0), (0, 1), (1, 1)):
            c = torch.full((M, N), 7.0, device="cuda")
            ctx.matmul_f32(a.T.contiguous() if ta else a, b.T.contiguous() if tb else b, c, M, K, N, trans_a=bool(ta), trans_b=bool(tb))
            ctx.finish()
            assert float(_row_errors(c, want).max()) <= _bound(K), (up, ta, tb)


@pytest.mark.parametrize("tokens,I,O", [(4096, 288, 320), (600, 64, 5000), (300, 64, 33000)])       # each block size of the split, and rows read twice
def test_partner_scales_of_a_weight_gradient(ctx, tokens, I, O):
    """dW whose largest contributions come from rows where x is small and grad_out large: the scale that completes x's row scales is
    not the one of the largest grad_out, and a sample that misses the row is put right."""
    state, scale, x, dy = _linear(tokens, I, O, 9)
    for row, dn, up in ((5, 40, 60), (tokens - 96, 60, 40), (177, 0, 30), (178, 100, 100)):
        x2, dy2 = x.clone(), dy.clone()
        x2[row] *= 2.0 ** -dn
        dy2[row, 11] *= 2.0 ** up
        for grouped in (0, 2):
            y, dx, dw, wy, wdx, wdw = _products(ctx, state, scale, x2, dy2, grouped)
            assert float((dw.double() - wdw).norm() / wdw.norm()) <= _bound(tokens)
            assert float(_row_errors(y, wy).max()) <= 1e-6 and float(_row_errors(dx, wdx).max()) <= 2.0 ** -22 + 2.0 ** -24 * 4 * (O / 64)


@pytest.mark.parametrize("K", [1, 7, 8, 9, 130, 252, 257, 4095, 4096, 4104, 10924, 32764, 32776, 40001])
@pytest.mark.parametrize("M", [1, 3, 1000])
def test_row_widths_of_the_split(ctx, M, K):
    """Chunks of many rows, of one row, rows wider than a chunk of either block size; rows of unequal magnitude; misaligned sources."""
    if M * K > 16_000_000:
        M = 300
    g = torch.Generator(device="cuda").manual_seed(K)
    N = 8
    buf = torch.randn(M * K + 1, device="cuda", generator=g)
    for off in (0, 1):
        a = buf[off:off + M * K].view(M, K)
        a.mul_(2.0 ** torch.randint(-30, 31, (M, 1), device="cuda", generator=g).float())
        b = torch.randn(N, K, device="cuda", generator=g)
        c, ct = torch.full((M, N), 7.0, device="cuda"), torch.full((N, M), 7.0, device="cuda")
        ctx.matmul_f32(a, b, c, M, K, N, trans_b=True)
        want = a.double() @ b.double().T
        size = a.double().abs() @ b.double().abs().T
        ctx.finish()
        assert float(((c.double() - want).norm(dim=1) / size.norm(dim=1)).max()) <= _bound(K)
        if M % 4 == 0:
            ctx.matmul_f32(b, a, ct, N, K, M, trans_b=True)           # the same rows as columns of the product
            ctx.finish()
            assert float(((ct.double().T - want).norm(dim=1) / size.norm(dim=1)).max()) <= _bound(K)
