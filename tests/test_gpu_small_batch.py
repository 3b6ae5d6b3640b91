"""Edges of the small-batch kernels that the shapes of test_gpu_skinny.py do not reach.

Tolerance, relative to max(|ref|, rms of the token's results): up to 16 tokens weights and activations enter exactly
(activations to 2^-22 of their record's largest for fp32), so what remains is fp32 accumulation inside a
record, at most 256 roundings of 2^-24 on sums a few times the result's rms: 1e-4.  Above 16 tokens fp32 activations
and Q6_K weights are rounded to fp16, 2^-11 each, and errors of K independent terms add up to about 2^-11 of the rms;
the largest of some thousand results is within a few times that: 2e-3.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import magnitude_b200 as mb  # noqa: E402

TYPES = [mb.TYPE_Q4_K, mb.TYPE_Q6_K, mb.TYPE_Q8_0, mb.TYPE_Q5_K, mb.TYPE_Q4_0, mb.TYPE_MXFP4]


def _weights(orc, backend, qt, n, k, seed):
    """Few distinct rows, so that a tall matrix is cheap to check: (handle, distinct rows dequantized, row of each)."""
    rng = np.random.default_rng(seed)
    base = orc.quantize(qt, rng.standard_normal((min(n, 96), k), dtype=np.float32) * np.float32(0.02))
    index = rng.integers(0, len(base), n)
    return backend.upload(qt, base[index], n, k), torch.from_numpy(orc.dequantize(qt, base, k)).cuda().double(), torch.from_numpy(index).cuda()


def _check(y, x, rows, index, rel):
    ref = (x.double() @ rows.T)[:, index]
    rms = ref.pow(2).mean(dim=1, keepdim=True).sqrt()
    worst = ((y.double() - ref).abs() / torch.maximum(ref.abs(), rms).clamp_min(1e-300)).max().item()
    assert worst <= rel, f"worst error {worst:.2e}"


# token tiles of 8, 16 and 32; tiles of 192 and 256 rows and one row more; whole, short and several chunks
@pytest.mark.parametrize("qt", TYPES)
@pytest.mark.parametrize("m", [3, 8, 9, 16, 17, 32])
@pytest.mark.parametrize("n,k", [(192, 256), (193, 2304), (257, 2048), (1025, 4352)])
def test_tile_edges(backend, orc, qt, m, n, k):
    w, rows, index = _weights(orc, backend, qt, n, k, n + m)
    x = torch.from_numpy(np.random.default_rng(m).standard_normal((m, k), dtype=np.float32)).cuda()
    for xx in (x.to(torch.bfloat16), x):
        y = backend.project(w, xx)
        backend.sync()
        _check(y, xx, rows, index, 1e-4 if m <= 16 else 2e-3)


# more slots per block than stages: prepared images, the ring goes round several times, tiles begin and end mid-block
@pytest.mark.parametrize("qt", TYPES)
@pytest.mark.parametrize("m", [7, 16, 31])
def test_many_slots_per_block(backend, orc, qt, m):
    w, rows, index = _weights(orc, backend, qt, 12289, 8448, m)
    x = torch.from_numpy(np.random.default_rng(m).standard_normal((m, 8448), dtype=np.float32)).cuda().to(torch.bfloat16)
    for _ in range(2):                       # the second run finds the shared tiles' sums and counts as the first left them
        y = backend.project(w, x)
        backend.sync()
        _check(y, x, rows, index, 1e-4 if m <= 16 else 2e-3)


# several weights of up to 48 rows run on these kernels, too; a single one only where it is large enough
@pytest.mark.parametrize("qt", TYPES)
@pytest.mark.parametrize("m", [20, 21, 33, 48, 49])
def test_sets_of_weights_up_to_48_rows(backend, orc, qt, m):
    shapes, k = [400, 193], 2304
    ws = [_weights(orc, backend, qt, n, k, n) for n in shapes]
    x = torch.from_numpy(np.random.default_rng(m).standard_normal((m, k), dtype=np.float32)).cuda()
    for xx in (x.to(torch.bfloat16), x):
        ys = backend.project_multi([w for w, _, _ in ws], xx)
        one = backend.project(ws[0][0], xx)
        backend.sync()
        for y, (_, rows, index) in zip(ys + [one], ws + [ws[0]]):
            _check(y, xx, rows, index, 2e-3)


# every record has a scale of its own: tokens of very different size, records of zeros, one channel far above the rest
@pytest.mark.parametrize("m", [8, 20])
def test_activation_range(backend, orc, m):
    k = 2048
    w, rows, index = _weights(orc, backend, mb.TYPE_Q4_K, 300, k, 1)
    x = torch.from_numpy(np.random.default_rng(2).standard_normal((m, k), dtype=np.float32)).cuda()
    x *= torch.exp2(torch.linspace(-60, 60, m, device="cuda"))[:, None]
    x[:, 256:512] = 0
    x[:, 700] *= 4096
    x[1] = 0
    x = x.to(torch.bfloat16)
    y = backend.project(w, x)
    backend.sync()
    _check(y, x, rows, index, 1e-4)          # bf16 tokens and Q4_K weights enter exactly at every batch size
    assert torch.all(y[1] == 0)


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_non_finite_activations_stay_in_their_token(backend, orc, value):
    w, rows, index = _weights(orc, backend, mb.TYPE_Q4_K, 300, 1024, 3)
    x = torch.from_numpy(np.random.default_rng(4).standard_normal((8, 1024), dtype=np.float32)).cuda().to(torch.bfloat16)
    x[5, 77] = value
    y = backend.project(w, x)
    backend.sync()
    assert not torch.isfinite(y[5]).any()
    keep = [0, 1, 2, 3, 4, 6, 7]
    _check(y[keep], x[keep], rows, index, 1e-4)


def test_a_product_has_the_same_bits_in_every_company(backend, orc):
    shapes = [(700, 4096), (2048, 4096), (513, 4096)]
    x = torch.from_numpy(np.random.default_rng(5).standard_normal((12, 4096), dtype=np.float32)).cuda().to(torch.bfloat16)
    ws = [_weights(orc, backend, mb.TYPE_Q5_K, n, k, i)[0] for i, (n, k) in enumerate(shapes)]
    alone = [backend.project(w, x) for w in ws]
    for _ in range(3):
        together = backend.project_multi(ws, x)
        backend.sync()
        for a, b in zip(alone, together):
            assert torch.equal(a, b)


# Host-buffer calls run on a stream of the library's own, which nothing orders after the calls in flight on the caller's:
# the two must not meet in a workspace.  Tiles shared by several blocks are the state that an overlap would spoil for good.
@pytest.mark.parametrize("m,m_host", [(8, 8), (16, 5), (20, 40), (300, 200)])
def test_host_calls_beside_device_calls(backend, orc, m, m_host):
    rel = 1e-4 if max(m, m_host) <= 16 else 2e-3
    w, rows, index = _weights(orc, backend, mb.TYPE_Q4_K, 1200, 8192, 6)
    h, hrows, hindex = _weights(orc, backend, mb.TYPE_Q6_K, 2100, 2304, 7)
    x = torch.from_numpy(np.random.default_rng(8).standard_normal((m, 8192), dtype=np.float32)).cuda()
    xh = np.random.default_rng(9).standard_normal((m_host, 2304), dtype=np.float32)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    out = [torch.empty((m, 1200), device="cuda") for _ in range(200)]
    for y in out:
        backend.project(w, x, out=y, stream=stream)
    hosts = [backend.project_host(h, xh) for _ in range(10)]
    backend.sync(stream)
    last = backend.project(w, x)
    backend.sync()
    for y in out + [last]:
        _check(y, x, rows, index, rel)
    for y in hosts:
        _check(torch.from_numpy(y).cuda(), torch.from_numpy(xh).cuda(), hrows, hindex, rel)


# A plan made after another one was destroyed may get the same addresses for other weights and images; run on a stream that is
# not ordered after anything its creation uploads.
@pytest.mark.parametrize("qt", [mb.TYPE_Q4_K, mb.TYPE_Q6_K])
def test_plans_made_and_destroyed_in_turn(backend, orc, qt):
    stream = torch.cuda.Stream()
    sets = []
    for k in (512, 2304, 4096):
        sets.append((k, [_weights(orc, backend, qt, 300 + 64 * i, k, k + i) for i in range(6)]))
    for turn in range(12):
        k, ws = sets[turn % 3]
        x = torch.from_numpy(np.random.default_rng(turn).standard_normal((6, k), dtype=np.float32)).cuda().to(torch.bfloat16)
        ys = [torch.empty((6, w.n), device="cuda") for w, _, _ in ws]
        torch.cuda.synchronize()
        plan = backend.plan([([w], x, [y]) for (w, _, _), y in zip(ws, ys)])
        plan.run(stream=stream)
        backend.sync(stream)
        for y, (_, rows, index) in zip(ys, ws):
            _check(y, x, rows, index, 1e-4)
        plan.close()


def _captured(call, warm):
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        warm()
    stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        call()
    return graph


@pytest.mark.parametrize("m,n", [(8, [640]), (16, [300, 1025]), (32, [640, 640])])
def test_replay_from_a_graph(backend, orc, m, n):
    k = 4352
    ws = [_weights(orc, backend, mb.TYPE_Q5_K, i, k, i) for i in n]
    x = torch.zeros((m, k), dtype=torch.bfloat16, device="cuda")
    ys = [torch.empty((m, i), device="cuda") for i in n]
    call = lambda: backend.project_multi([w for w, _, _ in ws], x, ys)      # noqa: E731
    graph = _captured(call, call)
    for turn in range(3):
        x.copy_(torch.from_numpy(np.random.default_rng(turn).standard_normal((m, k), dtype=np.float32)))
        graph.replay()
        backend.sync()
        for y, (_, rows, index) in zip(ys, ws):
            _check(y, x, rows, index, 1e-4 if m <= 16 else 2e-3)


# A set of 32 rows captured before the small-batch kernels' workspaces exist: a larger call has made what the GEMM needs
def test_capture_without_the_workspaces(orc):
    be = mb.Backend(0)
    k = 2048
    ws = [_weights(orc, be, mb.TYPE_Q4_K, n, k, n) for n in (400, 300)]
    x = torch.from_numpy(np.random.default_rng(1).standard_normal((100, k), dtype=np.float32)).cuda().to(torch.bfloat16)
    ys = [torch.zeros((32, n), device="cuda") for n in (400, 300)]
    graph = _captured(lambda: be.project_multi([w for w, _, _ in ws], x[:32], ys), lambda: be.project(ws[0][0], x))
    graph.replay()
    be.sync()
    for y, (_, rows, index) in zip(ys, ws):
        _check(y, x[:32], rows, index, 2e-3)
    del graph
    be.close()


# A plan owns its workspaces, 2.4 MB of sums per eight tokens (the driver hands out steps of 2 MB): they stay small beside a model's weights, also for an engine with two plans per layer
@pytest.mark.parametrize("m,limit_mb", [(4, 5), (16, 8)])
def test_memory_of_a_plan(backend, orc, m, limit_mb):
    w, _, _ = _weights(orc, backend, mb.TYPE_Q4_K, 512, 4096, 1)
    x = torch.zeros((m, 4096), dtype=torch.bfloat16, device="cuda")
    y = torch.empty((m, 512), device="cuda")
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    plans = [backend.plan([([w], x, [y])]) for _ in range(32)]
    used = (before - torch.cuda.mem_get_info()[0]) / 32 / 2**20
    for p in plans:
        p.close()
    assert used < limit_mb, f"{used:.1f} MB a plan"


# Plans share no state, so two of them may run at the same time
def test_two_plans_on_two_streams(backend, orc):
    made = []
    for seed, (qt, n, k, m) in enumerate([(mb.TYPE_Q4_K, 1300, 4096, 5), (mb.TYPE_Q6_K, 700, 8192, 12)]):
        ws = [_weights(orc, backend, qt, n + i, k, seed + i) for i in range(5)]
        x = torch.from_numpy(np.random.default_rng(seed).standard_normal((m, k), dtype=np.float32)).cuda().to(torch.bfloat16)
        ys = [torch.empty((m, w.n), device="cuda") for w, _, _ in ws]
        made.append((backend.plan([([w], x, [y]) for (w, _, _), y in zip(ws, ys)]), torch.cuda.Stream(), ws, x, ys))
    torch.cuda.synchronize()
    for _ in range(30):
        for plan, stream, _, _, _ in made:
            plan.run(stream=stream)
    for plan, stream, ws, x, ys in made:
        backend.sync(stream)
        for y, (_, rows, index) in zip(ys, ws):
            _check(y, x, rows, index, 1e-4)
        plan.close()


# A NaN must not come out as a number, whichever kernel takes the call: single weights and sets, 17 rows and more
@pytest.mark.parametrize("m,n", [(20, [300]), (32, [300]), (32, [300, 200]), (64, [300]), (150, [300]), (150, [40000])])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_nan_stays_nan_in_larger_batches(backend, orc, m, n, dtype):
    k = 1024
    ws = [_weights(orc, backend, mb.TYPE_Q4_K, i, k, i) for i in n]
    x = torch.from_numpy(np.random.default_rng(m).standard_normal((m, k), dtype=np.float32)).cuda().to(dtype)
    x[5, 77] = float("nan")
    ys = backend.project_multi([w for w, _, _ in ws], x)
    backend.sync()
    keep = [i for i in range(m) if i != 5]
    for y, (_, rows, index) in zip(ys, ws):
        assert torch.isnan(y[5]).all()
        _check(y[keep], x[keep], rows, index, 2e-3)


# Jobs of one plan may read one activation buffer with different K (and so need images of their own)
def test_plan_jobs_of_different_k_share_a_buffer(backend, orc):
    x = torch.from_numpy(np.random.default_rng(1).standard_normal((9, 4096), dtype=np.float32)).cuda().to(torch.bfloat16)
    ws = [_weights(orc, backend, mb.TYPE_Q8_0, n, k, n) for n, k in [(300, 4096), (257, 2048), (500, 4096), (193, 2304), (64, 2048)]]
    ys = [torch.empty((9, w.n), device="cuda") for w, _, _ in ws]
    plan = backend.plan([([w], x[:, :w.k], [y]) for (w, _, _), y in zip(ws, ys)])
    for _ in range(2):
        plan.run()
    backend.sync()
    for y, (w, rows, index) in zip(ys, ws):
        _check(y, x[:, :w.k], rows, index, 1e-4)
    plan.close()


# 16 tiles of 56 records: 144 blocks could share them, 128 with seven records each are as quick
@pytest.mark.parametrize("qt", [mb.TYPE_Q4_K, mb.TYPE_Q6_K])
@pytest.mark.parametrize("m", [8, 16, 20])
def test_equal_runs_of_records(backend, orc, qt, m):
    w, rows, index = _weights(orc, backend, qt, 3841, 14336, m)
    x = torch.from_numpy(np.random.default_rng(m).standard_normal((m, 14336), dtype=np.float32)).cuda().to(torch.bfloat16)
    for _ in range(2):
        y = backend.project(w, x)
        backend.sync()
        _check(y, x, rows, index, 1e-4 if m <= 16 else 2e-3)
