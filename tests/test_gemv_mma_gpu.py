"""Ternary GEMV of up to eight activation rows: clusters that split a row's chunks, 32-row units, recorded chains."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _matrix(rng, O, I):
    words = rng.integers(0, 2 ** 32, size=(O, I // 16), dtype=np.uint64).astype(np.uint32)
    digits = np.zeros((O, I), np.float64)
    for k in range(16):
        digits[:, k::16] = ((words >> np.uint32(2 * k)) & np.uint32(3)).astype(np.float64) - 1.0
    return torch.from_numpy(words.view(np.int32)).to(DEV), digits, rng.uniform(0.02, 0.2, O).astype(np.float32)


def _context():
    from motifcl_b200 import Context
    stream = torch.cuda.Stream(device=0)
    with torch.cuda.stream(stream):
        return stream, Context.on_torch_stream(0)


@pytest.mark.parametrize("M", [1, 2, 3, 5, 6, 7, 8])
@pytest.mark.parametrize("O,I", [(1, 64), (31, 256), (33, 320), (130, 1984), (257, 2112), (600, 14336), (9000, 512), (20001, 768)])
def test_edges_of_chunks_units_and_clusters(M, O, I):
    rng = np.random.default_rng(O * 31 + I + M)
    w, digits, scale = _matrix(rng, O, I)
    x = (rng.standard_normal((M, I)) * 10.0 ** rng.integers(-6, 6, (M, 1))).astype(np.float32)
    stream, ctx = _context()
    with torch.cuda.stream(stream):
        y = torch.full((M, O), 5.0, device=DEV)
        ctx.ternary_gemv(torch.from_numpy(x).to(DEV), w, torch.from_numpy(scale).to(DEV), y, M, I, O)
        got = y.cpu().numpy()
    want = x.astype(np.float64) @ digits.T * scale.astype(np.float64)
    size = np.abs(x.astype(np.float64)) @ np.abs(digits).T * scale.astype(np.float64)      # a sum of a few terms may cancel
    for m in range(M):
        assert np.linalg.norm(got[m] - want[m]) <= 1e-6 * np.linalg.norm(size[m])


@pytest.mark.parametrize("M", [1, 4, 8])
def test_recorded_chain_reads_the_result_before_it(M):
    """Recorded launches overlap: x of every second matrix is the result of the first, whose buffers the next pair takes again."""
    rng = np.random.default_rng(M)
    D, H = 1088, 4160
    up, up_d, up_s = _matrix(rng, H, D)
    down, down_d, down_s = _matrix(rng, D, H)
    x = rng.standard_normal((M, D)).astype(np.float32)
    stream, ctx = _context()
    with torch.cuda.stream(stream):
        us, ds = torch.from_numpy(up_s * 0.02).to(DEV), torch.from_numpy(down_s * 0.02).to(DEV)
        a, b = torch.from_numpy(x).to(DEV), torch.zeros(M, H, device=DEV)
        ctx.finish()
        ctx.batch_begin()
        for _ in range(6):
            ctx.ternary_gemv(a, up, us, b, M, D, H)
            ctx.ternary_gemv(b, down, ds, a, M, H, D)
        batch = ctx.batch_end()
        batch.launch()
        got = a.cpu().numpy()
        batch.close()
    want = x.astype(np.float64)
    for _ in range(6):
        want = (want @ up_d.T * us.cpu().numpy()) @ down_d.T * ds.cpu().numpy()
    assert np.linalg.norm(got - want) <= 1e-5 * np.linalg.norm(want)


def test_lane_recorded_again_reads_words_made_just_before():
    """A lane that ended an earlier recording with a GEMV: in the next recording the words are the result of the kernel before it,
    whatever handles the destroyed recording's nodes leave behind."""
    rng = np.random.default_rng(5)
    O, I, M = 8192, 4096, 2
    old, _, scale = _matrix(rng, O, I)
    state = torch.from_numpy(rng.integers(0, 256, O * I // 4 * 3, dtype=np.uint8)).to(DEV)
    x = rng.standard_normal((M, I)).astype(np.float32)
    stream, ctx = _context()
    from motifcl_b200 import Context
    with torch.cuda.stream(stream):
        lane = Context(0)
        sc, dx, y = torch.from_numpy(scale).to(DEV), torch.from_numpy(x).to(DEV), torch.empty(M, O, device=DEV)
        words, w = torch.empty_like(old), torch.empty(O, I, device=DEV)
        ctx.counter_decode_weight(state, sc, w, I, O, 11)
        want = dx.double() @ w.double().T
        ctx.finish()
        for _ in range(4):
            ctx.batch_begin()
            ctx.lane_fork(lane)
            for _ in range(2):
                lane.ternary_gemv(dx, old, sc, y, M, I, O)
            ctx.lane_join(lane)
            ctx.batch_end().close()
            ctx.batch_begin()
            ctx.lane_fork(lane)
            lane.counter_pack2(state, words, I, O, 11)
            lane.ternary_gemv(dx, words, sc, y, M, I, O)
            ctx.lane_join(lane)
            batch = ctx.batch_end()
            words.zero_()
            batch.launch()
            ctx.finish()
            batch.close()
            assert float((y.double() - want).norm() / want.norm()) <= 1e-6
        lane.close()
