"""The two-launch GEMM (fp16 copy of the weights, then a dense product) against the one-launch kernels.

Both dequantize with the same code and add up K in the same order on the tensor cores, so their results
are the same bits; the one-launch kernels are themselves held to the oracle in test_gpu_gemm.py.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import magnitude_b200 as mb  # noqa: E402

TYPES = [mb.TYPE_Q4_K, mb.TYPE_Q6_K, mb.TYPE_Q8_0, mb.TYPE_Q5_K, mb.TYPE_Q4_0, mb.TYPE_MXFP4]


def _backend(rows):
    """B200Q_GEMM_DENSE: 0 = one-launch kernels only, m = two launches from m rows on, unset = by estimate."""
    import os

    os.environ["B200Q_GEMM_DENSE"] = rows
    try:
        return mb.Backend(0)
    finally:
        del os.environ["B200Q_GEMM_DENSE"]


@pytest.fixture(scope="module")
def pair(backend):
    a, b = _backend("128"), _backend("0")
    yield a, b, backend
    a.close()
    b.close()


def _all(pair, qt, shapes, k, x, dtype):
    rng = np.random.default_rng(k + len(shapes))
    outs = []
    packed = []
    for n in shapes:
        base = mb.quantize(qt, rng.standard_normal((min(n, 64), k), dtype=np.float32) * np.float32(0.02))
        packed.append(base[rng.integers(0, len(base), n)])
    for be in pair:
        w = [be.upload(qt, p, n, k) for p, n in zip(packed, shapes)]
        y = [torch.full((x.shape[0], n + 8), 7.0, dtype=dtype, device="cuda")[:, :n] for n in shapes]
        be.project_multi(w, x, y) if len(w) > 1 else be.project(w[0], x, out=y[0])
        be.sync()
        outs.append(y)
        for v, n in zip(y, shapes):
            assert torch.all(torch.as_strided(v, (x.shape[0], 8), v.stride(), n) == 7.0)     # nothing past a row
    for a, b, c in zip(*outs):
        assert torch.equal(a, b) and torch.equal(a, c)


# edges of the 256-row stripes, the 32-token widths and the 8-record chunks; 512 tokens of 2560 rows: a last round of 20
# tiles of 256 tokens, cut into three of 96, 96 and 64
@pytest.mark.parametrize("qt", TYPES)
@pytest.mark.parametrize("m,shapes,k", [(128, [256], 256), (129, [257], 2304), (255, [511, 4, 130], 2048), (513, [1000], 4352), (512, [2560], 1024), (333, [2051, 260], 1280)])
def test_same_bits(pair, qt, m, shapes, k):
    x = torch.from_numpy(np.random.default_rng(m).standard_normal((m, k), dtype=np.float32)).cuda()
    _all(pair, qt, shapes, k, x.to(torch.bfloat16), torch.float32)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_activations_without_vector_access(pair, dtype):
    m, k = 200, 768
    buf = torch.from_numpy(np.random.default_rng(1).standard_normal((m, k + 3), dtype=np.float32)).cuda().to(dtype)
    _all(pair, mb.TYPE_Q4_K, [300], k, buf[:, 1:k + 1], torch.bfloat16)


def test_ragged_k(pair):
    x = torch.from_numpy(np.random.default_rng(2).standard_normal((140, 288), dtype=np.float32)).cuda().to(torch.bfloat16)
    _all(pair, mb.TYPE_Q8_0, [300], 288, x, torch.float32)


def test_weights_larger_than_the_workspace(pair):
    # 2 x 164 MB of fp16: two panels, the first ends in the second weight
    x = torch.from_numpy(np.random.default_rng(3).standard_normal((160, 4096), dtype=np.float32)).cuda().to(torch.bfloat16)
    _all(pair, mb.TYPE_Q4_K, [20100, 21000], 4096, x, torch.bfloat16)
