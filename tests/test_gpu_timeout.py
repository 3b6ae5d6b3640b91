"""A bounded device wait that runs out: the kernel returns, b200q_sync reports Timeout, the context
stays usable.  The wait is made to run out on the host's terms (a peer that never posts: the second
"rank" is a context that simply does not call), with the wait limit set to 50 ms; nothing faults,
traps or hangs.  One GPU: the two contexts live on the same device and only one of them launches."""
import ctypes
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import magnitude_b200 as mb  # noqa: E402
from magnitude_b200 import _binding as B  # noqa: E402
from magnitude_b200 import ggml_quant as gq  # noqa: E402


def test_peer_exchange_times_out_and_the_context_survives(orc):
    a, b = mb.Backend(0), mb.Backend(0)
    try:
        bufs = [a.peer_buffer(), b.peer_buffer()]
        a.peer_attach_buffers(0, 2, bufs)
        b.peer_attach_buffers(1, 2, bufs)
        a.set_option(B.OPT_WAIT_LIMIT_MS, 50)
        y = torch.ones(4096, device="cuda")
        a.allreduce(y)                                   # rank 1 never posts its share
        with pytest.raises(mb.B200QError) as e:
            a.sync()
        assert e.value.status == B.ERR_TIMEOUT
        # the context is not poisoned: an ordinary product still runs and is right
        n, k = 64, 1024
        packed = gq.synth_weights(mb.TYPE_Q4_K, n, k, 1)
        w = a.upload(mb.TYPE_Q4_K, packed, n, k)
        x = torch.randn(1, k, device="cuda").to(torch.bfloat16)
        out = a.project(w, x)
        a.sync()
        ref = orc.matmul_exact(mb.TYPE_Q4_K, packed, n, k, x.float().cpu().numpy())
        assert orc.within_tolerance(out.cpu().numpy(), ref, 1e-3)[0]
        # the ranks' call counters no longer agree: further exchanges are refused until both re-attach
        with pytest.raises(mb.B200QError) as e:
            a.allreduce(y)
        assert e.value.status == B.ERR_STOPPED
        a.peer_detach()
        b.peer_detach()
        a.peer_attach_buffers(0, 1, [a.peer_buffer()])   # a world of one: the sum is the input
        a.allreduce(y)
        a.sync()
        a.peer_detach()
        w.close()
    finally:
        a.set_option(B.OPT_WAIT_LIMIT_MS, 2000)
        a.close()
        b.close()


def _sharded(be, qt, n, k, rank, m):
    """Rank `rank` of two's half of a row-parallel product: weight and activations."""
    rng = np.random.default_rng(10 * rank + qt)
    w = be.upload(qt, gq.synth_weights(qt, n, k, 3 + rank), n, k)
    return w, torch.from_numpy(rng.standard_normal((m, k), dtype=np.float32)).cuda().to(torch.bfloat16)


@pytest.mark.parametrize("qt", [mb.TYPE_Q4_K, mb.TYPE_Q6_K])
@pytest.mark.parametrize("m", [1, 2])
@pytest.mark.parametrize("waits", [False, True])
def test_plan_sums_of_two_ranks_one_after_the_other(qt, m, waits):
    """Both ranks of a plan that sums inside its launch, on one GPU and one at a time.  Rank 1 posts its shares and its waits for
    rank 0 run out: Timeout.  Rank 0 then finds rank 1's shares in its buffer and ends with the sums, in rank order.  After the
    failure rank 1's plan, alone in the world, gives its own products again, run after run: a plan whose jobs wait finds its
    completion counter at zero."""
    n, n2, k = 200, 3000, 1024
    ranks = [mb.Backend(0), mb.Backend(0)]
    try:
        bufs = [be.peer_buffer() for be in ranks]
        plans, outs, own = [], [], []
        for r, be in enumerate(ranks):
            w, x = _sharded(be, qt, n, k, r, m)
            w2, x2 = _sharded(be, qt, n2, k, r + 2, m)
            own.append([be.project(w, x), be.project(w2, x2)])
            be.sync()
            outs.append([torch.zeros((m, n), device="cuda"), torch.zeros((m, n2), device="cuda")])
            plans.append(be.plan([([w], x, outs[r][:1]), ([w2], x2, outs[r][1:])], waits=[False, waits], sum_ranks=[True, True]))
            be.peer_attach_buffers(r, 2, bufs)
        ranks[0].set_option(B.OPT_WAIT_LIMIT_MS, 50)
        plans[1].run()
        with pytest.raises(mb.B200QError) as e:
            ranks[1].sync()
        assert e.value.status == B.ERR_TIMEOUT
        # (where jobs wait, the blocks that gave up first leave later jobs out: their shares may be missing)
        if not waits:
            plans[0].run()
            ranks[0].sync()
            for got, a, b in zip(outs[0], *own):
                assert torch.equal(got, a + b)
        for r, be in enumerate(ranks):
            be.peer_detach()
        for r in (1, 0):
            for _ in range(3):
                for o in outs[r]:
                    o.zero_()
                plans[r].run()
                ranks[r].sync()
                for got, want in zip(outs[r], own[r]):
                    assert torch.equal(got, want)
    finally:
        ranks[0].set_option(B.OPT_WAIT_LIMIT_MS, 2000)
        for be in ranks:
            be.close()


def _words(cu, base):
    """A device buffer's 64-bit words: (address, words)."""
    start, size = ctypes.c_uint64(), ctypes.c_size_t()
    assert cu.cuMemGetAddressRange_v2(ctypes.byref(start), ctypes.byref(size), ctypes.c_uint64(base)) == 0
    out = np.zeros(size.value // 8, np.uint64)
    assert cu.cuMemcpyDtoH_v2(out.ctypes.data_as(ctypes.c_void_p), start, ctypes.c_size_t(size.value)) == 0
    return start.value, out


def test_waiting_for_the_launch_before_has_no_limit(orc):
    """A launch that starts early stands idle until the one before has ended, however long that takes: here its two waits for a
    peer, each within the limit, together beyond it.  The peer's shares are copied into the buffer by the host."""
    n, k, m = 4, 1024, 1
    cu = ctypes.CDLL("libcuda.so.1")
    a, b, c = mb.Backend(0), mb.Backend(0), mb.Backend(0)
    try:
        bufs = [a.peer_buffer(), b.peer_buffer()]
        plans, outs, own = [], [], []
        for r, be in enumerate((a, b)):
            jobs = [_sharded(be, mb.TYPE_Q4_K, n, k, r + 2 * i, m) for i in range(2)]
            own.append([be.project(w, x) for w, x in jobs])
            be.sync()
            outs.append([torch.zeros((m, n), device="cuda") for _ in range(2)])
            plans.append(be.plan([([w], x, [o]) for (w, x), o in zip(jobs, outs[r])], sum_ranks=[True, True]))
            be.peer_attach_buffers(r, 2, bufs)
        big, xb = _sharded(c, mb.TYPE_Q4_K, 8192, 8192, 5, m)      # more than a ring holds, so that its producers wait
        want, got = c.project(big, xb), torch.zeros((m, 8192), device="cuda")
        c.sync()
        # rank 1 alone: its shares of exchanges 1 and 2 land in rank 0's buffer, its own wait runs out
        a.set_option(B.OPT_WAIT_LIMIT_MS, 50)
        plans[1].run()
        with pytest.raises(mb.B200QError):
            b.sync()
        base, words = _words(cu, bufs[0])
        assert cu.cuMemsetD8_v2(ctypes.c_uint64(base), ctypes.c_ubyte(0), ctypes.c_size_t(8 * len(words))) == 0
        a.set_option(B.OPT_WAIT_LIMIT_MS, 1000)
        stream = torch.cuda.Stream()
        torch.cuda.synchronize()
        plans[0].run(stream=stream)
        c.project(big, xb, out=got, stream=stream)
        for exchange in (1, 2):
            time.sleep(0.6)
            shares = np.flatnonzero(words >> np.uint64(32) == exchange)
            assert len(shares) == m * n
            for i in shares:
                word = words[i:i + 1]
                assert cu.cuMemcpyHtoD_v2(ctypes.c_uint64(base + 8 * int(i)), word.ctypes.data_as(ctypes.c_void_p), ctypes.c_size_t(8)) == 0
        a.sync(stream)
        c.sync(stream)
        assert torch.equal(got, want)
        for o, y0, y1 in zip(outs[0], *own):
            assert torch.equal(o, y0 + y1)
        a.peer_detach()
        b.peer_detach()
    finally:
        a.set_option(B.OPT_WAIT_LIMIT_MS, 2000)
        for be in (a, b, c):
            be.close()


def test_option_ranges(backend):
    for opt, bad in ((B.OPT_WAIT_LIMIT_MS, 0), (B.OPT_WAIT_LIMIT_MS, 10**7), (B.OPT_TP_INIT_TIMEOUT_MS, 0)):
        with pytest.raises(mb.B200QError):
            backend.set_option(opt, bad)
    backend.set_option(B.OPT_TP_INIT_TIMEOUT_MS, 30000)
