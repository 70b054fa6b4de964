"""Ternary GEMV: clusters that split a row's chunks, 32-row units, tiles cut between CTAs, recorded chains and lists."""
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


@pytest.mark.parametrize("M", [1, 2, 3, 5, 6, 7, 8, 9, 13, 16])
@pytest.mark.parametrize("O,I", [(1, 64), (31, 256), (33, 320), (130, 1984), (257, 2112), (600, 14336), (9000, 512), (20001, 768), (128, 256), (129, 28672)])
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


@pytest.mark.parametrize("M", [1, 3, 8, 9, 16])
@pytest.mark.parametrize("O,I,n", [(300, 1088, 1), (4096, 4096, 8)])
def test_the_smallest_magnitudes_have_their_bits(M, O, I, n):
    """Rows of 2^-90 down to 2^-125 and, beside them, subnormal activations; scales that bring the results back."""
    rng = np.random.default_rng(M)
    w, digits, scale = _matrix(rng, O, I)
    x = (rng.uniform(-1, 1, (M, I)) * 2.0 ** np.linspace(-90, -125, M)[:, None]).astype(np.float32)
    x[:, ::7] *= np.float32(2.0 ** -6)
    scale *= np.float32(2.0 ** 100)
    stream, ctx = _context()
    with torch.cuda.stream(stream):
        dx, s = torch.from_numpy(x).to(DEV), torch.from_numpy(scale).to(DEV)
        ys = [torch.full((M, O), 5.0, device=DEV) for _ in range(n)]
        ctx.ternary_gemv(dx, w, s, ys[0], M, I, O)
        ctx.finish()
        ctx.batch_begin()
        for y in ys:
            ctx.ternary_gemv(dx, w, s, y, M, I, O)
        batch = ctx.batch_end()
        batch.launch()
        ctx.finish()
        batch.close()
        want = x.astype(np.float64) @ digits.T * scale.astype(np.float64)
        for m in range(M):
            assert np.linalg.norm(ys[-1].cpu().numpy()[m] - want[m]) <= 1e-6 * np.linalg.norm(want[m])


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


@pytest.mark.parametrize("M", [1, 2, 3, 6, 8, 9, 16])
@pytest.mark.parametrize("shapes", [
    [(196, 256), (133, 256), (1025, 256)],                                    # clusters of one
    [(4096, 2048), (131, 2048), (6000, 14336), (257, 2112), (4096, 2048)],     # several lengths in clusters of eight
    [(9000, 512), (640, 4096), (177, 512), (640, 4096), (130, 1024)],         # clusters of 2 and of 8: two launches
    [(140, 320)] * 70,                                                        # more than one launch holds
    [(14336, 4096), (2000, 4096)] * 2, [(4096, 7168), (2048, 7168)] * 2,     # long enough for the tcgen05 kernel
    [(300, 1024), (5000, 1280), (257, 7168), (1000, 768)] * 2,                # clusters that shrink: two slices to a CTA
    [(8200, 768), (4000, 1280)] * 12,                                         # of it, in slices of one chunk and of two
])
def test_independent_matrices_of_a_recording_share_launches(M, shapes):
    """As one launch each, bit for bit, whatever shares a launch: two xs per length, rounds that end inside a matrix and a ring, tiles
    and slices that a cut runs through."""
    rng = np.random.default_rng(M * 100 + len(shapes))
    stream, ctx = _context()
    with torch.cuda.stream(stream):
        # of two xs per length, one whose slices of K may lie further apart than 2^8
        xs = {(I, h): torch.from_numpy((rng.standard_normal((M, I)) * 2.0 ** -(h * rng.integers(4, 14) * (np.arange(I) * 3 // I) / 2)).astype(np.float32)).to(DEV)
              for _, I in shapes for h in (0, 1)}
        mats = [_matrix(rng, O, I)[::2] for O, I in shapes]
        mats = [(w, torch.from_numpy(s).to(DEV)) for w, s in mats]
        ys, single = [[torch.full((M, O), 5.0, device=DEV) for O, _ in shapes] for _ in range(2)]

        def sweep(out):
            for i, ((O, I), (w, s)) in enumerate(zip(shapes, mats)):
                ctx.ternary_gemv(xs[I, i & 1], w, s, out[i], M, I, O)
        sweep(single)
        ctx.finish()
        before = ctx.launch_count
        ctx.batch_begin()
        sweep(ys)
        batch = ctx.batch_end()
        batch.launch()
        ctx.finish()
        assert ctx.launch_count - before < len(shapes)
        batch.close()
    for a, b in zip(ys, single):
        assert torch.equal(a, b)


@pytest.mark.parametrize("M,per", [(2, 1), (12, 2)])
def test_recorded_matrices_that_depend_on_one_another_keep_their_order(M, per):
    """Products of one x share a launch; what reads their results, overwrites them or stands behind another kernel does not join it."""
    rng = np.random.default_rng(3)
    D, H = 2048, 4096
    stream, ctx = _context()
    with torch.cuda.stream(stream):
        x, a, b, c = [torch.from_numpy(rng.standard_normal((M, n)).astype(np.float32)).to(DEV) for n in (D, H, D, D)]
        up, down, square = [(lambda w, s: (w, torch.from_numpy(s * 0.02).to(DEV)))(*_matrix(rng, *s)[::2]) for s in ((H, D), (D, H), (D, D))]

        def calls():
            ctx.ternary_gemv(x, *up, a, M, D, H)
            ctx.ternary_gemv(x, *square, b, M, D, D)         # beside the first
            ctx.ternary_gemv(a, *down, c, M, H, D)           # reads the first
            ctx.ternary_gemv(c, *up, a, M, D, H)             # reads the third and overwrites what it read
            ctx.ternary_gemv(x, *square, c, M, D, D)         # overwrites what the fourth read
            ctx.eltwise(0, c, b, c, M * D)                   # c += b
            ctx.ternary_gemv(c, *square, b, M, D, D)
            ctx.ternary_gemv(x, *square, c, M, D, D)         # overwrites what the launch before it reads
        calls()
        want = [t.clone() for t in (a, b, c)]
        ctx.finish()
        before = ctx.launch_count
        ctx.batch_begin()
        calls()
        batch = ctx.batch_end()
        for _ in range(3):
            batch.launch()
        ctx.finish()
        assert (ctx.launch_count - before) == 3 * (6 * per + 1)
        for t, w in zip((a, b, c), want):
            assert torch.equal(t, w)
        batch.close()


@pytest.mark.parametrize("M,shapes", [(4, [(14336, 4096), (14336, 4096)]), (8, [(4096, 4096)] * 2), (3, [(9000, 512)] * 60), (12, [(4096, 4096)] * 2)])
@pytest.mark.parametrize("by", ["lane", "event"])
def test_work_beside_a_recorded_list_waits_for_its_matrices(M, shapes, by):
    """A lane, or another stream by an event, reads and overwrites the first result while further matrices are recorded that the first
    one's launch could take; the list then grows long enough for the other kernel."""
    from motifcl_b200 import Context
    rng = np.random.default_rng(M)
    stream, ctx = _context()
    side = torch.cuda.Stream(device=0)
    with torch.cuda.stream(stream):
        lane = Context(0) if by == "lane" else Context(0, side.cuda_stream)
        x = {I: torch.from_numpy(rng.standard_normal((M, I)).astype(np.float32)).to(DEV) for _, I in shapes}
        mats = [(lambda w, s: (w, torch.from_numpy(s).to(DEV)))(*_matrix(rng, O, I)[::2]) for O, I in shapes]
        ys, want = [[torch.full((M, O), 5.0, device=DEV) for O, _ in shapes] for _ in range(2)]
        seen = torch.zeros_like(ys[0])

        def call(out, i):
            O, I = shapes[i]
            ctx.ternary_gemv(x[I], *mats[i], out[i], M, I, O)
        for i in range(len(shapes)):
            call(want, i)
        ctx.finish()
        lane.finish()
        ctx.batch_begin()
        call(ys, 0)
        if by == "lane":
            ctx.lane_fork(lane)
        else:
            side.wait_event(stream.record_event())
        lane.eltwise(4, ys[0], None, seen, seen.numel(), 1.0)          # seen = y + 1
        lane.eltwise(3, ys[0], None, ys[0], seen.numel(), 2.0)         # y = 2 y
        for i in range(1, len(shapes)):
            call(ys, i)
        if by == "lane":
            ctx.lane_join(lane)
        else:
            stream.wait_event(side.record_event())
        batch = ctx.batch_end()
        for _ in range(3):
            for y in ys:
                y.fill_(7.0)
            batch.launch()
            ctx.finish()
            assert torch.allclose(seen, want[0] + 1.0, rtol=1e-6, atol=1e-5)
            assert torch.allclose(ys[0], 2.0 * want[0], rtol=1e-6, atol=1e-5)
            for y, w in zip(ys[1:], want[1:]):
                assert torch.allclose(y, w, rtol=1e-6, atol=1e-5)
        batch.close()
        lane.close()


@pytest.mark.parametrize("M", [1, 2, 3, 5, 8])
@pytest.mark.parametrize("O,I,n", [(4096, 4096, 1), (14336, 4096, 1), (14336, 4096, 3), (2048, 14336, 8)])
def test_a_large_activation_that_no_weight_takes_leaves_the_other_slices(M, O, I, n):
    """An activation of 1e6 whose weights are 0, alone in its slice of K, beside ones of 1e-4: alone and in a list, on either kernel."""
    rng = np.random.default_rng(M + n)
    mats = []
    for _ in range(n):
        w, digits, scale = _matrix(rng, O, I)
        words = w.cpu().numpy().view(np.uint32)
        words[:, I // 2 // 16] = words[:, I // 2 // 16] & ~np.uint32(3) | np.uint32(1)         # field 1: digit 0
        digits[:, I // 2] = 0.0
        mats.append((torch.from_numpy(words.view(np.int32)).to(DEV), digits, scale))
    x = (rng.standard_normal((M, I)) * 1e-4).astype(np.float32)
    x[:, I // 2:I // 2 + I // 8] = 0.0
    x[:, I // 2] = 1e6
    stream, ctx = _context()
    with torch.cuda.stream(stream):
        dx = torch.from_numpy(x).to(DEV)
        args = [(w, torch.from_numpy(s).to(DEV), torch.full((M, O), 5.0, device=DEV)) for w, _, s in mats]
        single = torch.empty(M, O, device=DEV)
        ctx.ternary_gemv(dx, *args[0][:2], single, M, I, O)
        ctx.finish()
        ctx.batch_begin()
        for w, s, y in args:
            ctx.ternary_gemv(dx, w, s, y, M, I, O)
        batch = ctx.batch_end()
        batch.launch()
        ctx.finish()
        batch.close()
        assert torch.equal(args[0][2], single)
        for (_, digits, scale), (_, _, y) in zip(mats, args):
            want = x.astype(np.float64) @ digits.T * scale.astype(np.float64)
            assert np.linalg.norm(y.cpu().numpy() - want) <= 1e-6 * np.linalg.norm(want)


@pytest.mark.parametrize("M", [1, 2, 8, 12, 16])
def test_lists_that_fill_the_gpu_with_tiles_of_two_accumulators(M):
    """10752 k-blocks: tiles of 256 rows, two CTAs on every SM, whatever the number of rows; ragged matrices, two xs, one of them (up to 8
    rows) in slices.  Two launches, against float64 and, bit for bit, against single calls, which up to 2 rows run on the other kernel."""
    rng = np.random.default_rng(M)
    shapes = [(14300, 4096), (4096, 14336), (13999, 4096), (4001, 14336), (14336, 4096), (14081, 4096)]
    stream, ctx = _context()
    with torch.cuda.stream(stream):
        g = torch.Generator(device=DEV).manual_seed(M)
        xs = {I: torch.randn(M, I, device=DEV, generator=g) for I in (4096, 14336)}
        xs[14336] *= 2.0 ** -(torch.arange(14336, device=DEV) * 3 // 14336 * 6).float()
        mats = [(torch.randint(-2 ** 31, 2 ** 31 - 1, (O, I // 16), dtype=torch.int32, device=DEV, generator=g),
                 torch.rand(O, device=DEV, generator=g) + 0.1) for O, I in shapes]
        ys, single = [[torch.full((M, O), 5.0, device=DEV) for O, _ in shapes] for _ in range(2)]

        def sweep(out):
            for (O, I), (w, s), y in zip(shapes, mats, out):
                ctx.ternary_gemv(xs[I], w, s, y, M, I, O)
        sweep(single)
        ctx.finish()
        before = ctx.launch_count
        ctx.batch_begin()
        sweep(ys)
        batch = ctx.batch_end()
        batch.launch()
        ctx.finish()
        assert ctx.launch_count - before == 2
        batch.close()
        for (O, I), (w, s), y, one in zip(shapes, mats, ys, single):
            assert torch.equal(y, one)
            digits = torch.stack([((w >> (2 * k)) & 3).double() - 1.0 for k in range(16)], dim=2).view(O, I)
            want = (xs[I].double() @ digits.T) * s.double()
            for m in range(M):
                assert float((y[m] - want[m]).norm() / want[m].norm()) <= 1e-6


@pytest.mark.parametrize("M", [9, 13, 16])
@pytest.mark.parametrize("O,I", [(4096, 4096), (4001, 14336), (130, 4160), (2000, 6144), (1024, 14336), (257, 2048), (14336, 4096)])
def test_one_matrix_whose_tiles_are_cut(M, O, I):
    """More than 8 rows: sums of a tile over a cluster of 2 to 8 CTAs or, where more share it, over the workspace; alone, as a chain of recorded
    launches, and as the first of a list that has grown."""
    rng = np.random.default_rng(O + I + M)
    w, digits, scale = _matrix(rng, O, I)
    x = rng.standard_normal((M, I)).astype(np.float32)
    want = x.astype(np.float64) @ digits.T * scale.astype(np.float64)
    stream, ctx = _context()
    with torch.cuda.stream(stream):
        dx, s = torch.from_numpy(x).to(DEV), torch.from_numpy(scale).to(DEV)
        one, chain, first, second = [torch.full((M, O), 5.0, device=DEV) for _ in range(4)]
        ctx.ternary_gemv(dx, w, s, one, M, I, O)
        ctx.finish()
        before = ctx.launch_count
        ctx.batch_begin()
        for _ in range(3):
            ctx.ternary_gemv(dx, w, s, chain, M, I, O)           # overwrites its own result: launches of their own
        batch = ctx.batch_end()
        ctx.batch_begin()
        ctx.ternary_gemv(dx, w, s, first, M, I, O)
        ctx.ternary_gemv(dx, w, s, second, M, I, O)
        pair = ctx.batch_end()
        for _ in range(2):
            batch.launch()
            pair.launch()
        ctx.finish()
        assert ctx.launch_count - before == 2 * (6 + 2)
        batch.close()
        pair.close()
        assert np.linalg.norm(one.cpu().numpy() - want) <= 1e-6 * np.linalg.norm(want)
        for y in (chain, first, second):
            assert torch.equal(y, one)


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("M,O,I", [(1, 4001, 44032), (2, 4001, 44032), (4, 4001, 44032), (6, 4001, 44032), (7, 4001, 14336), (8, 4001, 14336), (8, 2000, 28672)])
def test_one_matrix_of_up_to_eight_rows_whose_tiles_are_cut(M, O, I, wide):
    """Long enough for the tcgen05 kernel by itself: sums of a tile over a cluster, or over the workspace where x has to be taken in slices;
    alone and as a chain of recorded launches."""
    stream, ctx = _context()
    with torch.cuda.stream(stream):
        g = torch.Generator(device=DEV).manual_seed(M + I)
        x = torch.randn(M, I, device=DEV, generator=g)
        if wide:
            x *= 2.0 ** -(torch.arange(I, device=DEV) * 3 // I * 6).float()
        w = torch.randint(-2 ** 31, 2 ** 31 - 1, (O, I // 16), dtype=torch.int32, device=DEV, generator=g)
        s = torch.rand(O, device=DEV, generator=g) + 0.1
        one, chain = torch.full((M, O), 5.0, device=DEV), torch.full((M, O), 5.0, device=DEV)
        before = ctx.launch_count
        ctx.ternary_gemv(x, w, s, one, M, I, O)
        ctx.finish()
        ctx.batch_begin()
        for _ in range(2):
            ctx.ternary_gemv(x, w, s, chain, M, I, O)
        batch = ctx.batch_end()
        for _ in range(2):
            batch.launch()
        ctx.finish()
        assert ctx.launch_count - before == 2 * (1 + 4)
        batch.close()
        digits = torch.stack([((w >> (2 * k)) & 3).double() - 1.0 for k in range(16)], dim=2).view(O, I)
        want = (x.double() @ digits.T) * s.double()
        assert torch.equal(one, chain)
        for m in range(M):
            assert float((one[m] - want[m]).norm() / want[m].norm()) <= 1e-6
