"""Products of fp32 tensors whose magnitudes are spread: an element far above the others, wherever it lies, and the gradients of
a classifier.  Every product is compared with float64.  The bound: 2^-22 for the terms of both operands, and for each tensor-core
instruction that adds into one accumulator half a last bit of what it holds, 2^-24, because it truncates and one large term
may fill it from the start (at most 64 k-tiles of 64, three products of four instructions each)."""
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
