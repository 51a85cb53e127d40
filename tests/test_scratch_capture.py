"""Work space of streams and of captured calls: which is kept, which is given back, and results of graphs whatever else ran before their replay."""
import pytest
import torch


@pytest.fixture
def streams(monkeypatch):
    """Streams by number and whether they are being captured, without a GPU."""
    from bmtrain_b200.ops import gemm

    state = {"stream": 0, "capturing": False, "made": []}

    class Made:
        def __init__(self, index, stream):
            self.stream = stream
            state["made"].append(stream)

    monkeypatch.setattr(torch._C, "_cuda_getDevice", lambda: 0, raising=False)
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda index: state["stream"], raising=False)
    monkeypatch.setattr(torch._C, "_cuda_isCurrentStreamCapturing", lambda: state["capturing"], raising=False)
    monkeypatch.setattr(gemm, "_Scratch", Made)
    monkeypatch.setattr(gemm, "_scratch", {})
    monkeypatch.setattr(gemm, "_latest", (None, None), raising=False)
    return gemm, state


def test_streams_in_use_keep_their_scratch(streams):
    gemm, state = streams

    def on(stream):
        state["stream"] = stream
        return gemm.scratch()

    main = on(0)
    for stream in range(1, 3 * gemm._MOST_SCRATCH):
        assert on(stream).stream == stream
        assert on(0) is main                    # used all the time, so it is never the one that goes
        assert len(gemm._scratch) <= gemm._MOST_SCRATCH
    assert on(3 * gemm._MOST_SCRATCH - 1).stream == 3 * gemm._MOST_SCRATCH - 1
    assert len(state["made"]) == 3 * gemm._MOST_SCRATCH


def test_nothing_that_a_capture_made_is_kept(streams):
    gemm, state = streams
    state["capturing"] = True
    first, second = gemm.scratch(), gemm.scratch()
    assert first is not second and not state["made"] and not gemm._scratch
    assert tuple(first.gemm) == (0, 0)          # tiles stay whole
    state["capturing"] = False
    own = gemm.scratch()
    assert own is gemm.scratch() and state["made"] == [0]
    state["capturing"] = True
    assert gemm.scratch() is not own


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_captured_bias_gradients(bmt_gpu, dtype):
    from bmtrain_b200.ops import gemm as G

    gen = torch.Generator(device="cuda").manual_seed(2)
    g = torch.randn(3000, 520, generator=gen, device="cuda").to(dtype)
    h = torch.randn(2100, 1000, generator=gen, device="cuda").to(dtype)
    a = torch.randn(256, 10240, generator=gen, device="cuda").to(dtype)
    want = G.bias_grad(g), G.bias_grad(h), G.gemm_nt(a, a)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    graphs = [torch.cuda.CUDAGraph() for _ in range(2)]
    outs = []
    for graph in graphs:                        # the first use of the stream is in a capture
        with torch.cuda.graph(graph, stream=side):
            outs.append((G.bias_grad(g), G.bias_grad(h), G.gemm_nt(a, a)))

    def right(got):
        torch.cuda.synchronize()
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
        assert (got[2].double() - want[2].double()).norm() <= 2 * (2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8) * want[2].double().norm()

    with torch.cuda.stream(side):
        right((G.bias_grad(g), G.bias_grad(h), G.gemm_nt(a, a)))
    graphs[1].replay()                          # before the first one
    right(outs[1])
    for _ in range(2 * G._MOST_SCRATCH):        # streams come and go
        with torch.cuda.stream(torch.cuda.Stream()):
            right((G.bias_grad(g), G.bias_grad(h), G.gemm_nt(a, a)))
    junk = [torch.full((1 << 20,), 77, dtype=torch.int32, device="cuda") for _ in range(64)]
    for graph, out in zip(graphs, outs):
        for t in out:
            t.zero_()
        graph.replay()
        right(out)
    assert all(bool((j == 77).all()) for j in junk)


@pytest.mark.gpu
def test_captured_block_backward(bmt_gpu):
    """A block of more tokens than one column-sum kernel walks over, captured forward and backward, against the same calls outside."""
    from bmtrain_b200.ops import gpt_block

    gen = torch.Generator(device="cuda").manual_seed(4)
    d, f, tokens = 256, 512, 2200
    rnd = lambda *s: 0.05 * torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    shapes = [(d,), (d,), (3 * d, d), (3 * d,), (d, d), (d,), (d,), (d,), (f, d), (f,), (d, f), (d,)]
    params = [((1 if i in (0, 6) else 0) + rnd(*s)).half() for i, s in enumerate(shapes)]
    x, dy = rnd(1, tokens, d).half(), rnd(1, tokens, d).half()

    def step(grads):
        run = gpt_block.Pass(x, None, [p.data_ptr() for p in params], 4, 64, f, "relu", 1e-5, True)
        return run.forward(), run.backward(dy, [t.data_ptr() for t in grads])

    want = [torch.empty_like(p) for p in params]
    y, dx = step(want)
    got = [torch.empty_like(p) for p in params]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = step(got)
    for _ in range(2):
        for t in got:
            t.zero_()
        graph.replay()
        torch.cuda.synchronize()
        # tiles that are divided outside of a capture are added in another order there; a dozen 16-bit intermediates follow one another
        for a, e in [(captured[0], y), (captured[1], dx)] + list(zip(got, want)):
            assert (a.double() - e.double()).norm() <= 12 * 2.0 ** -11 * e.double().norm()
