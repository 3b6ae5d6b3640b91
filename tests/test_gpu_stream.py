"""The streaming kernel's rules: ring sizes (and with them the number of teams), row quads that are not full, last chunks
of every length, parts of the grid for plans of small products.  A result never depends on any of them."""
import ctypes
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import magnitude_b200 as mb  # noqa: E402

TYPES = [mb.TYPE_Q4_K, mb.TYPE_Q5_K, mb.TYPE_Q6_K, mb.TYPE_Q8_0, mb.TYPE_Q4_0, mb.TYPE_MXFP4]
REL = 1e-3      # the decode route's bound: activations in 16-bit fixed point, seen 7e-5


def _weights(orc, qt, n, k, seed):
    return orc.quantize(qt, np.random.default_rng(seed).standard_normal((n, k), dtype=np.float32) * np.float32(0.02))


def _acts(m, k, seed):
    return torch.from_numpy(np.random.default_rng(seed).standard_normal((m, k), dtype=np.float32)).cuda().to(torch.bfloat16)


@pytest.mark.parametrize("qt", TYPES)
@pytest.mark.parametrize("m,n,k", [(1, 1, 256), (1, 2367, 256 * 9), (2, 17, 256 * 11), (1, 700, 256 * 20), (2, 4700, 256 * 7), (1, 13, 256 * 33), (2, 1184, 2304), (1, 1185, 2304)])
def test_rows_and_chunks_of_every_length(backend, orc, qt, m, n, k):
    """(Up to 1184 rows, two row groups a block, run on the form without second rows.)"""
    p = _weights(orc, qt, n, k, n + k)
    x = _acts(m, k, 3)
    y = backend.project(backend.upload(qt, p, n, k), x)
    backend.sync()
    assert backend.last_route()[0] == mb.ROUTE_GEMV
    ref = orc.matmul_exact(qt, p, n, k, x.float().cpu().numpy())
    assert orc.within_tolerance(y.cpu().numpy(), ref, REL)[0]


@pytest.mark.parametrize("qt", TYPES)
@pytest.mark.parametrize("peak,weight", [(2e-34, 1.0), (1e-33, 1.0), (9e37, 0.005), (1e38, 0.005), (2e38, 0.005), (2.9e38, 0.005)])
@pytest.mark.parametrize("m", [1, 2])
def test_blocks_of_extreme_size(backend, orc, qt, peak, weight, m):
    """Every 32-element block's largest magnitude is `peak`: near the ends of what the fixed-point step's quotient can hold.
    Calls, and a plan of two jobs (activations converted by a launch of their own), fp32 and bf16."""
    n, k = 70, 1024
    p = orc.quantize(qt, np.random.default_rng(qt).standard_normal((n, k), dtype=np.float32) * np.float32(weight))
    w = backend.upload(qt, p, n, k)
    rng = np.random.default_rng(9)
    x = rng.uniform(-1, 1, (m, k)).astype(np.float32)
    x[:, ::32] = rng.choice(np.float32([-1, 1]), (m, k // 32))
    x = torch.from_numpy(x * np.float32(peak)).cuda()
    for a in (x, x.to(torch.bfloat16)):
        y, y1, y2 = backend.project(w, a), torch.zeros((m, n), device="cuda"), torch.zeros((m, n), device="cuda")
        plan = backend.plan([([w], a, [y1]), ([w], a, [y2])])
        plan.run()
        backend.sync()
        assert orc.within_tolerance(y.cpu().numpy(), orc.matmul_exact(qt, p, n, k, a.float().cpu().numpy()), REL)[0]
        assert torch.equal(y1, y) and torch.equal(y2, y)


@pytest.mark.parametrize("qt", [mb.TYPE_Q4_K, mb.TYPE_Q6_K, mb.TYPE_Q8_0])
@pytest.mark.parametrize("m", [1, 2])
def test_results_do_not_depend_on_the_ring(backend, orc, qt, m):
    """From all of the shared memory down to what is refused, in steps smaller than a slot and then smaller than a copy of the
    partial sums: every number of slots and teams down to one, and one copy of the sums.  Two to three row quads a block, a
    final pass after each; calls, plans of independent jobs and one with a job that waits, whose
    activation is converted in the launch between two prepared ones."""
    n, k = 3000, 256 * 65
    p, p2 = _weights(orc, qt, n, k, 1), _weights(orc, qt, 300, 2304, 2)
    x, x2 = _acts(m, k, 5), _acts(m, 2304, 6)
    ref, limit, step, accepted = None, 232448, 8192, 0
    while True:
        os.environ["B200Q_GEMV_SMEM"] = str(limit)
        be = mb.Backend(0)
        os.environ.pop("B200Q_GEMV_SMEM", None)
        w, w2 = be.upload(qt, p, n, k), be.upload(qt, p2, 300, 2304)
        out = [torch.zeros((m, n), device="cuda") for _ in range(3)] + [torch.zeros((m, 300), device="cuda") for _ in range(2)]
        try:
            out.append(be.project(w, x))
            for o, waits in ((out[0:2] + out[3:4], [False, True, False]), ([out[2], torch.zeros_like(out[2]), out[4]], None)):
                plan = be.plan([([w], x, o[:1]), ([w2], x2, o[2:]), ([w], x, o[1:2])], waits=waits)
                for _ in range(2):
                    plan.run()
                be.sync()
                assert torch.equal(o[0], o[1])
        except mb.B200QError:
            be.close()
            if step == 1024:
                break
            limit, step = limit + step - 1024, 1024
            continue
        if ref is None:
            ref = out
            assert orc.within_tolerance(out[0].cpu().numpy(), orc.matmul_exact(qt, p, n, k, x.float().cpu().numpy()), REL)[0]
            assert orc.within_tolerance(out[3].cpu().numpy(), orc.matmul_exact(qt, p2, 300, 2304, x2.float().cpu().numpy()), REL)[0]
        for a, b in zip(out, ref):
            assert torch.equal(a, b), limit
        assert torch.equal(out[0], out[2]) and torch.equal(out[0], out[5]) and torch.equal(out[3], out[4])
        be.close()
        accepted += 1
        limit -= step
    assert step == 1024 and accepted >= 8


@pytest.mark.parametrize("m", [1, 2])
def test_plans_of_small_products_share_the_grid(backend, orc, m):
    """Products of few rows run on halves and quarters of the grid, beside a large one and a SWIGLU job; three runs alike.
    (Which part a job gets: test_stream_rules.py.)"""
    shapes = [(mb.TYPE_Q4_K, 512, 1024), (mb.TYPE_Q4_K, 1000, 4096), (mb.TYPE_Q6_K, 37, 512), (mb.TYPE_Q8_0, 4096, 4096), (mb.TYPE_Q4_K, 14336, 4096)]
    shapes = (shapes * 5)[:23]
    jobs, outs, want = [], [], []
    for i, (qt, n, k) in enumerate(shapes):
        w = backend.upload(qt, _weights(orc, qt, n, k, i % 5), n, k)
        x = _acts(m, k, i)
        y = torch.zeros((m, n), device="cuda")
        jobs.append(([w], x, [y]))
        outs.append(y)
        want.append(backend.project(w, x))
    g, u = jobs[0][0][0], backend.upload(mb.TYPE_Q4_K, _weights(orc, mb.TYPE_Q4_K, 512, 1024, 99), 512, 1024)
    act = torch.zeros((m, 512), device="cuda")
    gate, up = want[0].double(), backend.project(u, jobs[0][1]).double()
    for extra in (False, True):
        plan = backend.plan(jobs + ([([g, u], jobs[0][1], [act])] if extra else []), **({"swiglu": [False] * len(jobs) + [True]} if extra else {}))
        for _ in range(3):
            for y in outs + [act]:
                y.zero_()
            plan.run()
            backend.sync()
            for a, b in zip(outs, want):
                assert torch.equal(a, b)
            if extra:       # the quick exponential: a few units in the last place, and a division and a product
                assert torch.allclose(act.double(), gate / (1 + torch.exp(-gate)) * up, rtol=2e-6, atol=1e-12)


@pytest.mark.parametrize("qt", [mb.TYPE_Q4_K, mb.TYPE_Q4_0, mb.TYPE_MXFP4])
@pytest.mark.parametrize("m,k", [(1, 84992), (2, 42496), (4, 21248)])
def test_rows_that_fill_the_shared_memory(backend, orc, qt, m, k):
    """The longest activations that fit beside one ring slot, where the partial sums have one copy: calls, and jobs that wait and
    add to what is there."""
    n = 41 * 4 + 3
    p = _weights(orc, qt, n, k, 4)
    w, x = backend.upload(qt, p, n, k), _acts(m, k, 7)
    ref = orc.matmul_exact(qt, p, n, k, x.float().cpu().numpy())
    if m <= 2:
        y = backend.project(w, x)
        backend.sync()
        assert orc.within_tolerance(y.cpu().numpy(), ref, REL)[0]
    y = torch.zeros((m, n), device="cuda")
    plan = backend.plan([([w], x, [y])] * 2, waits=[False, True], accumulate=[True, True])
    plan.run()
    backend.sync()
    assert orc.within_tolerance(y.cpu().numpy(), 2 * ref, REL)[0]


def _edge_types(graph):
    """Types of a captured graph's edges: 0 ordinary, 1 programmatic (the later launch may start before the earlier has ended)."""
    cu, count = ctypes.CDLL("libcuda.so.1"), ctypes.c_size_t(8)
    nodes, data = (ctypes.c_void_p * 8)(), (ctypes.c_uint8 * 64)()
    assert cu.cuGraphGetEdges_v2(ctypes.c_void_p(graph.raw_cuda_graph()), nodes, (ctypes.c_void_p * 8)(), data, ctypes.byref(count)) == 0
    return [data[8 * i + 2] for i in range(count.value)]


def test_only_independent_plans_start_before_the_launch_before_has_ended(backend, orc):
    """A launch whose jobs wait holds SMs until all its blocks run, so it may not come in beside another stream's."""
    n, k = 64, 512
    w = backend.upload(mb.TYPE_Q4_K, _weights(orc, mb.TYPE_Q4_K, n, k, 1), n, k)
    x, y = _acts(1, k, 2), [torch.zeros((1, n), device="cuda") for _ in range(2)]
    for waits in (False, True):
        plan = backend.plan([([w], x, [y[0]]), ([w], x, [y[1]])], waits=[False, waits])
        graph = torch.cuda.CUDAGraph(keep_graph=True)
        with torch.cuda.graph(graph):
            plan.run()
        assert _edge_types(graph) == [0 if waits else 1]       # activation preparation -> products
