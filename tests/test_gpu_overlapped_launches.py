"""Kernels that may start before the stream's previous kernel has ended: a long
producer ahead of a call, a consumer that rewrites its input behind it, and calls
that read what the call before wrote, on one stream with no synchronisation, several
times over.  Every result has to be the one of the same call by itself."""
import pytest

pytestmark = pytest.mark.gpu
N = 300_007
FORMS = [(6, "--hamming_window"), (7, "--hanning_window --remove_dc"), (8, "--layout=dense"),
         (9, "--hamming_window"), (10, "--hanning_window --remove_dc"), (11, "--half_complex_return"),
         (12, "--hamming_window"), (12, "--half_complex_return"), (13, "--layout=dense"),
         (14, "--hanning_window"), (15, "--half_complex_return --layout=dense"), (16, "--hamming_window"),
         (17, "--remove_dc"), (18, "--half_complex_return"), (19, "--hamming_window"), (20, "--hamming_window")]
ROUNDS = 6


def _sources(torch):
    g = torch.Generator(device="cuda").manual_seed(5)
    return [torch.randn(N, generator=g, device="cuda") for _ in range(ROUNDS)]


def _overlap(torch, src, call, want, results):
    """call() reads `x`; results() are the buffers it writes."""
    x, run = call
    for s, w in zip(src, want):
        x.copy_(s)
        torch.cuda.synchronize()
        run()
        torch.cuda.synchronize()
        w[:] = [r.clone() for r in results]
    big = torch.zeros(1 << 26, device="cuda")
    got = []
    torch.cuda.synchronize()
    for s in src:
        big.add_(1.0)  # some 80 us of work ahead of the producer
        x.copy_(s)
        run()
        got.append([r.clone() for r in results])
        x.fill_(float("nan"))
    torch.cuda.synchronize()
    for i, (g, w) in enumerate(zip(got, want)):
        for a, b in zip(g, w):
            assert torch.equal(a, b), i


@pytest.mark.parametrize("exp,opts", FORMS)
def test_producer_and_consumer(ocs_lib, monkeypatch, exp, opts):
    import torch

    monkeypatch.setenv("OCS_AUTOTUNE", "0")
    src = _sources(torch)
    g = ocs_lib.geometry(N, exp, 0.5, opts)
    x, out = torch.zeros(N, device="cuda"), torch.zeros(g.out_floats, device="cuda")
    # a second request reads the first one's result
    n2 = min(N, g.out_floats)
    g2 = ocs_lib.geometry(n2, exp, 0.3, opts)
    out2 = torch.zeros(g2.out_floats, device="cuda")

    def run():
        ocs_lib.activate_device(x, N, exp, 0.5, opts, out, g.out_floats)
        ocs_lib.activate_device(out, n2, exp, 0.3, opts, out2, g2.out_floats)

    _overlap(torch, src, (x, run), [[] for _ in src], [out, out2])


@pytest.mark.parametrize("count", [3, 60])
def test_batches(ocs_lib, monkeypatch, count):
    """Batches of every window: one launch for all (few requests) and one per class."""
    import torch

    monkeypatch.setenv("OCS_AUTOTUNE", "0")
    src = _sources(torch)
    x = torch.zeros(N, device="cuda")
    opts = ["--hamming_window", "--half_complex_return", "--hanning_window --serial_power", "--layout=dense"]
    items = []
    for i in range(count):
        e, o = 6 + i % 8, opts[i % 4]
        g = ocs_lib.geometry(N, e, 0.5, o)
        items.append((x, N, e, 0.5, o, torch.zeros(g.out_floats, device="cuda"), g.out_floats))
    reqs = ocs_lib.make_requests(items)
    _overlap(torch, src, (x, lambda: ocs_lib.batch_device(reqs)), [[] for _ in src], [it[5] for it in items])


@pytest.mark.parametrize("exp", [6, 10, 13, 16])
def test_stage_hooks(ocs_lib, exp):
    import torch

    rf = ocs_lib.runnerFunction
    src = _sources(torch)
    g = ocs_lib.geometry(N, exp, 0.5, "")
    x = torch.zeros(N, device="cuda")
    re, im, out = (torch.zeros(g.ofull, device="cuda") for _ in range(3))

    def run():
        rf.Overlap(x, g.ofull, N, exp, g.hop, re)
        rf.Window("Hanning", re, g.ofull, g.n_window)
        rf.RemoveDC(re, g.qt, g.ofull, g.n_window)
        rf.EXP(re, im, g.ohalf, exp)
        rf.ToPower(out, re, im, g.ofull)

    _overlap(torch, src, (x, run), [[] for _ in src], [out, re, im])


@pytest.mark.parametrize("exp", [10, 13, 16, 18, 20])
def test_captured_calls(ocs_lib, monkeypatch, exp):
    """The same edges inside a graph, where the long windows' scratch is the graph's own."""
    import torch

    monkeypatch.setenv("OCS_AUTOTUNE", "0")
    src = _sources(torch)
    g = ocs_lib.geometry(N, exp, 0.5, "")
    x, out, out2 = (torch.zeros(k, device="cuda") for k in (N, g.out_floats, g.out_floats))
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()

    def call(o):
        ocs_lib.activate_device(x, N, exp, 0.5, "", o, g.out_floats)

    call(out)  # plans and tables
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        with torch.cuda.graph(graph, stream=stream):
            call(out)
            call(out2)
    _overlap(torch, src, (x, graph.replay), [[] for _ in src], [out, out2])
    call(out)
    x.copy_(src[0])
    call(out)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, out2)
