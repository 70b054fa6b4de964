"""The workspace of a context: who takes it, and whose addresses inside it outlive its growth."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
DEV = "cuda:0"
I = O = 1152


def _context():
    from motifcl_b200 import Context
    stream = torch.cuda.Stream(device=0)
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        return stream, Context.on_torch_stream(0)


class _Forward:
    """A product whose operands' terms lie in the workspace; 16 times the tokens need a larger one."""

    def __init__(self, seed):
        g = torch.Generator(device=DEV).manual_seed(seed)
        self.state = torch.randint(0, 256, (O * I // 4 * 3,), dtype=torch.uint8, device=DEV, generator=g)
        self.scale = torch.rand(O, device=DEV, generator=g) + 0.1
        self.x = torch.randn(4096, I, device=DEV, generator=g)
        self.y = torch.empty(4096, O, device=DEV)
        torch.cuda.synchronize()

    def small(self, ctx):
        ctx.counter_forward(self.x, self.state, self.scale, self.y, 256, I, O, 11)

    def grow(self, ctx):
        """...and write over whatever memory became free."""
        before = ctx.workspace_bytes
        ctx.counter_forward(self.x, self.state, self.scale, self.y, 4096, I, O, 11)
        ctx.finish()
        assert ctx.workspace_bytes > before
        torch.empty(1 << 28, device=DEV).fill_(float("nan"))
        torch.cuda.synchronize()
        self.y.fill_(5.0)
        torch.cuda.synchronize()

    def eager(self, ctx):
        self.small(ctx)
        ctx.finish()
        return self.y[:256].clone()


def _words(rng, rows, cols):
    return torch.from_numpy(rng.integers(0, 2 ** 32, size=(rows, cols // 16), dtype=np.uint64).astype(np.uint32).view(np.int32)).to(DEV)


def test_growth_keeps_what_a_graph_of_the_caller_holds():
    stream, ctx = _context()
    f = _Forward(1)
    with torch.cuda.stream(stream):
        want = f.eager(ctx)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
            f.small(ctx)
        f.grow(ctx)
        graph.replay()
        ctx.finish()
        assert torch.equal(f.y[:256], want)
        del graph
        ctx.close()


def test_growth_of_a_lane_keeps_what_a_batch_holds():
    from motifcl_b200 import Context
    stream, ctx = _context()
    f = _Forward(2)
    with torch.cuda.stream(stream):
        lane = Context(0)
        want = f.eager(lane)
        ctx.batch_begin()
        ctx.lane_fork(lane)
        f.small(lane)
        ctx.lane_join(lane)
        batch = ctx.batch_end()
        f.grow(lane)
        batch.launch()
        ctx.finish()
        assert torch.equal(f.y[:256], want)
        batch.close()
        lane.close()
        ctx.close()


@pytest.mark.parametrize("M", [1, 2, 4, 8])
def test_decode_of_up_to_eight_rows_does_without(M):
    """Alone and where the caller captures the stream (there also a matrix that rather takes workspace)."""
    rng = np.random.default_rng(M)
    stream, ctx = _context()
    with torch.cuda.stream(stream):
        for rows, cols, eager in ((1024, 4096, True), (14336, 4096, False)):
            w, scale = _words(rng, rows, cols), torch.full((rows,), 0.05, device=DEV)
            x, y = torch.randn(M, cols, device=DEV), torch.empty(M, rows, device=DEV)
            stream.synchronize()
            if eager:
                ctx.ternary_gemv(x, w, scale, y, M, cols, rows)
                ctx.finish()
                assert ctx.workspace_bytes == 0
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
                ctx.ternary_gemv(x, w, scale, y, M, cols, rows)
            assert ctx.workspace_bytes == 0
            y.fill_(5.0)
            graph.replay()
            stream.synchronize()
            got = y.clone()
            del graph
            ctx.ternary_gemv(x, w, scale, y, M, cols, rows)
            ctx.finish()
            assert torch.equal(got, y)
            if eager:
                assert ctx.workspace_bytes == 0
        ctx.close()


@pytest.mark.parametrize("on", ["context", "lane"])
def test_lists_of_a_recording_get_workspace_beside_a_batch_that_holds_some(on):
    from motifcl_b200 import Context
    rng = np.random.default_rng(7)
    stream, ctx = _context()
    f = _Forward(3)
    M, rows, cols, n = 8, 4096, 4096, 12
    with torch.cuda.stream(stream):
        who = ctx if on == "context" else Context(0)
        want = f.eager(who)

        def recorded(calls):
            ctx.batch_begin()
            if who is not ctx:
                ctx.lane_fork(who)
            calls()
            if who is not ctx:
                ctx.lane_join(who)
            return ctx.batch_end()
        first = recorded(lambda: f.small(who))
        mats = [_words(rng, rows, cols) for _ in range(n)]
        scale, x = torch.full((rows,), 0.05, device=DEV), torch.randn(M, cols, device=DEV)
        ys, single = [[torch.full((M, rows), 5.0, device=DEV) for _ in mats] for _ in range(2)]
        stream.synchronize()
        before = who.workspace_bytes

        def sweep(out):
            for w, y in zip(mats, out):
                who.ternary_gemv(x, w, scale, y, M, cols, rows)
        sweep(single)
        who.finish()
        assert who.workspace_bytes == before
        second = recorded(lambda: sweep(ys))
        assert who.workspace_bytes > before
        torch.empty(1 << 28, device=DEV).fill_(float("nan"))
        f.y.fill_(5.0)
        for _ in range(2):
            first.launch()
            second.launch()
        ctx.finish()
        assert torch.equal(f.y[:256], want)
        for a, b in zip(ys, single):
            assert torch.equal(a, b)
        first.close()
        second.close()
        if who is not ctx:
            who.close()
        ctx.close()


def test_growth_that_fails_leaves_the_workspace():
    """A call whose terms no device can hold (its sizes are refused before anything is read)."""
    from motifcl_b200 import MotifclCudaError
    stream, ctx = _context()
    f = _Forward(4)
    with torch.cuda.stream(stream):
        want = f.eager(ctx)
        before = ctx.workspace_bytes
        with pytest.raises(MotifclCudaError, match="workspace allocation"):
            ctx.counter_forward(f.x, f.state, f.scale, f.y, 1 << 29, I, O, 11)
        assert ctx.workspace_bytes == before
        f.y.fill_(5.0)
        assert torch.equal(f.eager(ctx), want)
        ctx.close()
