"""Kernels whose launches overlap the ones before them in their stream: chains
of dependent calls enqueued back to back give what the same calls give with
the device idle between them, on a context's own stream, on the caller's, and
captured into a graph and replayed."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
P = (1 << 31) - 1


@pytest.fixture(scope="module")
def B():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from gpustark.backend import GpuBackend
    return GpuBackend


def chain(B, cols, log, tw, idle, ctx=None, out=None):
    """Interpolate in place, extend by 2, hash the rows, build the tree."""
    def step():
        if idle:
            torch.cuda.synchronize()
    new = lambda words: torch.empty(words, dtype=torch.int32, device="cuda")
    ev = out[0] if out else [new(1 << (log + 1)) for _ in cols]
    layers = out[1] if out else [new(8 << k) for k in range(log + 2)]
    B.interpolate_columns(cols, log, tw, ctx=ctx)
    step()
    B.evaluate_polynomials(cols, log + 1, tw, ctx=ctx, out=ev)
    step()
    B.commit_on_layer(log + 1, None, ev, ctx=ctx, out=layers[-1])
    step()
    B.commit_node_layers(layers, ctx=ctx)
    step()
    return ev, layers


def columns(log, n, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return list(torch.randint(0, P, (n, 1 << log), dtype=torch.int32, device="cuda", generator=g))


@pytest.mark.parametrize("log,n", [(5, 3), (9, 16), (13, 5), (14, 40), (17, 33)])
def test_back_to_back_equals_one_at_a_time(B, log, n):
    tw = B.precompute_twiddles(log)
    for seed in range(8):
        a, b = columns(log, n, seed), columns(log, n, seed)
        ev, layers = chain(B, a, log, tw, idle=False)
        ev1, layers1 = chain(B, b, log, tw, idle=True)
        assert all(torch.equal(x, y) for x, y in zip(a + ev + layers, b + ev1 + layers1))


def test_captured_and_replayed(B):
    from gpustark.backend import Context
    log, n = 14, 24
    tw = B.precompute_twiddles(log)
    fresh = columns(log, n, 3)
    want = chain(B, columns(log, n, 3), log, tw, idle=True)
    s = torch.cuda.Stream()
    ctx = Context(s)
    cols = list(torch.zeros(n, 1 << log, dtype=torch.int32, device="cuda"))
    out = (list(torch.zeros(n, 2 << log, dtype=torch.int32, device="cuda")),
           [torch.zeros(8 << k, dtype=torch.int32, device="cuda") for k in range(log + 2)])
    torch.cuda.synchronize()
    chain(B, cols, log, tw, idle=False, ctx=ctx, out=out)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        chain(B, cols, log, tw, idle=False, ctx=ctx, out=out)
    for _ in range(3):
        for c, f in zip(cols, fresh):
            c.copy_(f)
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(out[0] + out[1], want[0] + want[1]))


@pytest.mark.parametrize("log,n,off", [(6, 3, 1), (13, 20, 1), (18, 4, 0), (18, 4, 1)])
def test_layers_right_behind_the_kernels_they_read(B, log, n, off):
    """Layers of a thread per node, over columns and children that the kernels
    before them in the stream write."""
    tw = B.precompute_twiddles(log)
    for seed in range(4):
        got = []
        for idle in (False, True):
            rows = torch.stack(columns(log, n, seed))
            mem = torch.zeros(n, (1 << log) + 4, dtype=torch.int32, device="cuda")
            cols = [r[off:off + (1 << log)] for r in mem]
            mem[:, off:off + (1 << log)] = rows
            kids = torch.zeros(16 << log, dtype=torch.int32, device="cuda")
            torch.cuda.synchronize()
            B.interpolate_columns(cols, log, tw)
            B.commit_on_layer(log + 1, None, [torch.cat([c, c]) for c in cols], out=kids)
            if idle:
                torch.cuda.synchronize()
            layer = B.commit_on_layer(log, kids, cols)
            if idle:
                torch.cuda.synchronize()
            got.append(B.commit_on_layer(log - 1, layer, []))
        assert torch.equal(*got)
