"""A bounded device-side wait that runs out: the kernel returns, the status block says where, the context lives on.

``nq_row_reduce_p2p`` polls its inbox for the words its peers push.  Here it is called as rank 0 of a group of
two whose second member does not exist: ``inbox[1]`` is a second allocation on the same GPU that nobody reads
and no kernel ever pushes into ``inbox[0]``, so the poll can only end by its time limit (set to 2 ms for the
test).  Nothing faults, traps or spins without bound; the call must complete, report
``NQ_ERR_DEVICE_TIMEOUT`` with the site of the wait, and leave the device usable.
"""
import ctypes
import time

import pytest
import torch

pytestmark = pytest.mark.gpu

NQ_ERR_DEVICE_TIMEOUT = -5
SITE_ROW_REDUCE = 64
SITE_PRODUCER, SITE_MMA_FULL, SITE_MMA_TMEM_EMPTY, SITE_EPI_TMEM_FULL, SITE_SCALE_FULL, SITE_SCALE_EMPTY = 1, 2, 3, 4, 5, 6
SITE_WEIGHT_LANE = 16


@pytest.fixture(scope="module")
def lib(built_library):
    from nano_qwen_b200 import _cabi, ops
    ops.init()
    return _cabi.lib()


def test_row_reduce_poll_gives_up_and_reports(lib):
    from nano_qwen_b200 import _cabi, ops
    from oracle import fp8_spec as S
    torch.cuda.synchronize()
    assert _cabi.device_status(reset=True)["code"] in (0, NQ_ERR_DEVICE_TIMEOUT)
    slot = 4096
    ptrs = []

    def alloc(nbytes):
        p = ctypes.c_void_p()
        _cabi.check(lib.nq_p2p_alloc(nbytes, ctypes.byref(p)), "nq_p2p_alloc")
        ptrs.append(p)
        return p.value

    try:
        mine, absent_peer, state = alloc(2 * 2 * 2 * slot), alloc(2 * 2 * 2 * slot), alloc(256)
        inbox = (ctypes.c_void_p * 2)(mine, absent_peer)
        y = torch.ones(1024, dtype=torch.bfloat16, device="cuda")
        _cabi.check(lib.nq_set_wait_limit_ns(2_000_000), "nq_set_wait_limit_ns")
        t0 = time.perf_counter()
        st = lib.nq_row_reduce_p2p(y.data_ptr(), y.data_ptr(), y.numel(), inbox, 0, 2, slot, state,
                                   torch.cuda.current_stream().cuda_stream)
        assert st == 0                                     # the call itself is accepted and enqueued
        torch.cuda.synchronize()                           # ... and it ends, although no peer ever answers
        waited = time.perf_counter() - t0
        assert waited < 1.0, f"the poll should give up after about 2 ms, took {waited:.3f} s"
        status = _cabi.device_status()
        assert status["code"] == NQ_ERR_DEVICE_TIMEOUT
        assert status["where"] == SITE_ROW_REDUCE and status["aux"] == 1        # waiting for rank 1
        with pytest.raises(_cabi.NqError):
            ops.check_device_status()                      # what a host loop calls at its synchronisation points
    finally:
        lib.nq_set_wait_limit_ns(2_000_000_000)
        _cabi.device_status(reset=True)
        torch.cuda.synchronize()
        for p in ptrs:
            lib.nq_p2p_free(p)
    # the device and the library are still usable: an ordinary linear passes against the oracle
    g = torch.Generator().manual_seed(3)
    x = torch.randn(40, 512, generator=g).to(torch.bfloat16)
    w = (torch.randn(256, 512, generator=g) * 0.02).to(torch.bfloat16)
    wq, sw = S.quantize_weight_block128(w)
    yy = ops.fp8_linear(x.cuda(), wq.cuda(), sw.cuda())
    torch.cuda.synchronize()
    xq, sx = S.quantize_act_group128(x)
    assert S.max_rel_err(yy.cpu(), S.linear_dequant_matmul(xq, sx, wq, sw)) <= 2e-2
    assert _cabi.device_status()["code"] == 0
    ops.check_device_status()


class AbsentPeer:
    """A reduction of two ranks whose second member does not exist: it occupies the stream for as long as its wait limit."""

    def __init__(self, lib):
        from nano_qwen_b200 import _cabi
        self.lib, self.slot, self.ptrs = lib, 4096, []
        for nbytes in (16 * self.slot, 16 * self.slot, 256):
            p = ctypes.c_void_p()
            _cabi.check(lib.nq_p2p_alloc(nbytes, ctypes.byref(p)), "nq_p2p_alloc")
            self.ptrs.append(p)
        self.inbox = (ctypes.c_void_p * 2)(self.ptrs[0].value, self.ptrs[1].value)
        self.y = torch.ones(1024, dtype=torch.bfloat16, device="cuda")

    def occupy_stream(self, ms: float):
        assert self.lib.nq_set_wait_limit_ns(int(ms * 1e6)) == 0
        assert self.lib.nq_row_reduce_p2p(self.y.data_ptr(), self.y.data_ptr(), self.y.numel(), self.inbox, 0, 2, self.slot,
                                          self.ptrs[2], torch.cuda.current_stream().cuda_stream) == 0

    def free(self):
        self.lib.nq_set_wait_limit_ns(2_000_000_000)
        torch.cuda.synchronize()
        for p in self.ptrs:
            self.lib.nq_p2p_free(p)


@pytest.fixture
def absent_peer(lib):
    from nano_qwen_b200 import _cabi
    torch.cuda.synchronize()
    _cabi.device_status(reset=True)
    peer = AbsentPeer(lib)
    yield peer
    peer.free()
    _cabi.device_status(reset=True)


def quantised(m, n, k, seed):
    from oracle import fp8_spec as S
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(m, k, generator=g).to(torch.bfloat16)
    w = (torch.randn(n, k, generator=g) * 0.02).to(torch.bfloat16)
    return x, S.quantize_act_group128(x), S.quantize_weight_block128(w)


def decode_gemm_behind_a_waiting_reduction(lib, peer, case, algo, split_k):
    """The GEMM starts beside the reduction, 60 ms long, and requests its weights; its activations may be read when the
    reduction has ended, but its issuing and epilogue threads wait 2 ms only.  Returns y (a sentinel where nothing was
    stored) and the time that the two launches took."""
    from nano_qwen_b200 import ops
    x, (xq, sx), (wq, sw) = case
    x, xq, sx, wq, sw = x.cuda(), xq.cuda(), sx.t().contiguous().cuda().t(), wq.cuda(), sw.cuda()
    y = torch.full((x.shape[0], wq.shape[0]), -777.0, dtype=torch.bfloat16, device="cuda")
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    peer.occupy_stream(60)
    assert lib.nq_set_wait_limit_ns(2_000_000) == 0
    if algo == ops.ALGO_WEIGHT_LANE_FUSED:
        ops.fp8_linear(x, wq, sw, out=y, algo=algo, split_k=split_k)
    else:
        ops.fp8_gemm(xq, sx, wq, sw, out=y, algo=algo, split_k=split_k)
    lib.nq_set_wait_limit_ns(2_000_000_000)
    torch.cuda.synchronize()
    return y.cpu(), time.perf_counter() - t0


@pytest.mark.parametrize("algo,m,split_k", [("WEIGHT_LANE", 8, 8), ("WEIGHT_LANE", 8, 1), ("WEIGHT_LANE", 24, 4),
                                            ("WEIGHT_LANE", 64, 8), ("WEIGHT_LANE", 100, 8), ("WEIGHT_LANE", 200, 8),
                                            ("WEIGHT_LANE_FUSED", 8, 8), ("WEIGHT_LANE_FUSED", 32, 1)])
def test_decode_gemm_gives_up_with_copies_still_to_come(lib, absent_peer, algo, m, split_k):
    """With 8 splits a CTA's whole K range fits its ring: the producer never waits for a stage, it requests the activations
    after the other roles have given up, and the CTA must not end before they have landed.  With one split the ring goes
    round: scale loader and quantisers find stages that nobody has read and must leave them alone.  The same call then passes."""
    from nano_qwen_b200 import _cabi, ops
    from oracle import fp8_spec as S
    case = quantised(m, 512, 4096, m + split_k)
    y, waited = decode_gemm_behind_a_waiting_reduction(lib, absent_peer, case, getattr(ops, "ALGO_" + algo), split_k)
    status = _cabi.device_status(reset=True)
    assert status["code"] == NQ_ERR_DEVICE_TIMEOUT
    # the issuer's or the epilogue's first wait, at once (the reduction's own limit expires 58 ms later); the fused kernel's
    # producer waits for nothing else than its first stage, to which it comes back after the fifth K-tile
    first = [(4096 // 128) * z // split_k for z in range(split_k)]
    expired = (status["where"] - SITE_WEIGHT_LANE, status["aux"])
    assert expired[0] in (SITE_MMA_FULL, SITE_EPI_TMEM_FULL) and expired[1] in first or (
        algo == "WEIGHT_LANE_FUSED" and expired[0] == SITE_PRODUCER and expired[1] - 5 in first), expired
    assert bool((y == -777.0).all()) and waited < 1.0               # every CTA gave up
    x, (xq, sx), (wq, sw) = case
    y = ops.fp8_gemm(xq.cuda(), sx.cuda(), wq.cuda(), sw.cuda(), algo=ops.ALGO_WEIGHT_LANE, split_k=split_k)
    torch.cuda.synchronize()
    assert S.max_rel_err(y.cpu(), S.linear_dequant_matmul(xq, sx, wq, sw)) <= 2e-2
    assert _cabi.device_status()["code"] == 0


@pytest.mark.parametrize("algo", ["TOKEN_LANE_128", "TOKEN_LANE_192", "TOKEN_LANE_256", "TOKEN_PAIR"])
@pytest.mark.parametrize("k", [128, 384])
def test_persistent_gemm_gives_up_and_stores_no_wrong_value(lib, algo, k):
    """Rows of y with an odd stride are stored element by element: 20 to 45 us for a tile, in which the other roles wait for
    accumulators, stages and scale blocks.  A limit of 1 ns lets each wait probe its barrier twice (8 us), so they give up.
    The launch ends with the status of a timeout; an element of y has its value or was left alone."""
    from nano_qwen_b200 import _cabi, ops
    torch.cuda.synchronize()
    _cabi.device_status(reset=True)
    m, n, which = 4096, 4096, getattr(ops, "ALGO_" + algo)
    gen = torch.Generator(device="cuda").manual_seed(k)
    xq, sx = ops.act_quant(torch.randn(m, k, generator=gen, device="cuda").to(torch.bfloat16))
    wq, sw = ops.weight_quant(torch.randn(n, k, generator=gen, device="cuda").to(torch.bfloat16))
    wide = torch.full((m, n + 1), -777.0, dtype=torch.bfloat16, device="cuda")
    want = ops.fp8_gemm(xq, sx, wq, sw, algo=which)
    torch.cuda.synchronize()
    assert _cabi.device_status()["code"] == 0
    try:
        assert lib.nq_set_wait_limit_ns(1) == 0
        t0 = time.perf_counter()
        ops.fp8_gemm(xq, sx, wq, sw, out=wide[:, 1:], algo=which)
        torch.cuda.synchronize()
        waited = time.perf_counter() - t0
    finally:
        lib.nq_set_wait_limit_ns(2_000_000_000)
    status = _cabi.device_status(reset=True)
    assert status["code"] == NQ_ERR_DEVICE_TIMEOUT and waited < 0.5
    assert status["where"] in (SITE_PRODUCER, SITE_MMA_FULL, SITE_MMA_TMEM_EMPTY, SITE_EPI_TMEM_FULL, SITE_SCALE_FULL, SITE_SCALE_EMPTY)
    assert 0 <= status["aux"] < k // 128 and 0 <= status["block"] < 148
    left = wide[:, 1:] == -777.0
    assert bool(left.any()) and bool((left | (wide[:, 1:] == want)).all()) and bool((wide[:, 0] == -777.0).all())
    ops.fp8_gemm(xq, sx, wq, sw, out=wide[:, 1:], algo=which)
    torch.cuda.synchronize()
    assert torch.equal(wide[:, 1:], want) and _cabi.device_status()["code"] == 0
