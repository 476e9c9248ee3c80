"""What a call reports: non-finite coefficients and factors end in the documented error, at every place where they
could get lost (one chunk, a chunk edge, several chunks), and leave the context usable."""

import pytest
import torch

import oal_b200

pytestmark = pytest.mark.gpu

BAD = [float("nan"), float("inf"), -float("inf")]
ERROR = "denominator must be finite and strictly positive"


def _inputs(n, g, hq=4, hkv=2):
    gen = torch.Generator().manual_seed(n + g)
    q, k, v = (torch.randn(1, h, n, 64, generator=gen).bfloat16().cuda() for h in (hq, hkv, hkv))
    groups = (torch.arange(64) % g).to(torch.int32).cuda()
    return q, k, v, groups


# the per-head factorisation of explicit coefficients orders its terms by sign: a NaN has none
@pytest.mark.parametrize("n", [64, 128, 129, 300])
@pytest.mark.parametrize("g", [1, 8, 16])
@pytest.mark.parametrize("value", BAD)
def test_non_finite_explicit_coefficients_raise(n, g, value):
    q, k, v, groups = _inputs(n, g)
    for which in range(3):
        coefs = [torch.ones(4), torch.ones(4, g), torch.eye(g).expand(4, g, g).clone()]
        coefs[which].view(4, -1)[1, -1] = value
        with pytest.raises(RuntimeError, match=ERROR):
            oal_b200.grouped_coefficient_attention(q, k, v, groups, *(c.cuda() for c in coefs), precision="bf16_tensorcore")
    coefs = [torch.ones(4), torch.ones(4, g), torch.eye(g).expand(4, g, g).clone()]
    out, _, _ = oal_b200.grouped_coefficient_attention(q, k, v, groups, *(c.cuda() for c in coefs), precision="bf16_tensorcore")
    assert torch.isfinite(out).all()


# a factor that is not finite: the one-call form, a prepared inference and training call, a recorded step
@pytest.mark.parametrize("n", [1, 64, 128, 129, 300])
@pytest.mark.parametrize("g", [1, 8, 16])
@pytest.mark.parametrize("value", BAD)
def test_non_finite_factors_raise(n, g, value):
    from oal_b200 import hd_block_gemm_autograd as hd
    from oal_b200.captured_step import CapturedStep

    q, k, v, groups = _inputs(n, g)
    good = torch.full((4, (g + 1) * (g + 2) // 2), 0.5, device="cuda")
    for entry in (0, 1, good.shape[1] - 1):
        factor = good.clone()
        factor[1, entry] = value
        with pytest.raises(RuntimeError, match=ERROR):
            oal_b200.oal_attention(q, k, v, groups, factor)
        prepared = oal_b200.prepare_grouped_hd_block_gemm(q, k, v, groups, good, precision="bf16_tensorcore")
        with pytest.raises(RuntimeError, match=ERROR):
            oal_b200.run_prepared_grouped_hd_block_gemm(prepared, q, k, v, factor)
        leaves = [t.clone().requires_grad_() for t in (q, k, v, factor)]
        prepared = oal_b200.prepare_grouped_hd_block_gemm(*leaves[:3], groups, leaves[3], precision="bf16_tensorcore")
        with pytest.raises(RuntimeError, match=ERROR):
            oal_b200.run_prepared_grouped_hd_block_gemm(prepared, *leaves)[0].sum().backward()
            hd.check_pending_status(block=True)
    leaves = [t.clone().requires_grad_() for t in (q, k, v, good)]
    prepared = oal_b200.prepare_grouped_hd_block_gemm(*leaves[:3], groups, leaves[3], precision="bf16_tensorcore")
    step = CapturedStep(prepared, *leaves, torch.ones_like(leaves[0]))
    step.replay(*(t.detach() for t in leaves), torch.ones_like(q))
    step.check_status()
    step.replay(q, k, v, factor, torch.ones_like(q))
    with pytest.raises(RuntimeError, match=ERROR):
        step.check_status()
    hd.forget_captured_status()


# one chunk (prologue alone), several (prologue in the state update's launch, its rotations beside it or in it)
@pytest.mark.parametrize("n", [100, 300, 1000])
@pytest.mark.parametrize("overlap", [1, 0])
def test_packed_forward_owns_its_status_words(n, overlap):
    """Status words and workspace hold anything before the call; a clean call leaves zero, delivers it and counts no
    word of an earlier one."""
    import ctypes

    from oal_b200 import _lib
    from oal_b200.hd_block_gemm import make_problem
    from oal_b200.hd_block_gemm_autograd import build_group_tables

    lib = _lib.load()
    q, k, v, groups = _inputs(n, 8)
    tables = build_group_tables(groups.expand(4, -1), 8)
    factor = torch.full((4, 45), 0.5, device="cuda")
    problem = make_problem((1, 4, 2, n, 64, 64), groups=8, io_dtype=torch.bfloat16, out_dtype=torch.bfloat16,
                           precision="bf16_tensorcore", chunk=128, scale=0.125, floor=1e-38, flags=_lib.FLAG_ZERO_STATE_IN)
    out, num, den = torch.empty_like(q), torch.empty(q.shape, device="cuda"), torch.empty(q.shape[:3], device="cuda")
    ws, saved = (torch.full((_lib.workspace_bytes(problem, phase),), 255, dtype=torch.uint8, device="cuda") for phase in (0, 2))
    coefs, status = torch.empty(4 * 73, device="cuda"), torch.full((2,), 0x55555555, dtype=torch.int32, device="cuda")
    ticket, word = ctypes.c_int64(0), ctypes.c_int32(-1)
    torch.cuda.synchronize()
    lib.oal_set_overlap(overlap)
    try:
        _lib.check(lib.oal_forward_packed(
            ctypes.byref(problem), *(_lib.ptr(t) for t in (q, k, v, tables.dim_perm, tables.group_start, factor)), 4, 1e-6,
            *(_lib.ptr(t) for t in (coefs, out, num, den, saved, ws)), ws.numel(), _lib.ptr(status), ctypes.byref(ticket),
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        assert lib.oal_status_poll(ticket.value, 1, ctypes.byref(word)) == 1 and word.value == 0
    finally:
        lib.oal_set_overlap(1)
    torch.cuda.synchronize()
    assert status[0].item() == 0 and torch.isfinite(out).all()
    want = oal_b200.oal_attention(q, k, v, groups, factor, scale=0.125)
    assert torch.equal(out, want)


SLEEP = 1_000_000_000      # clocks of torch.cuda._sleep: about half a second


def _warm(prepared, *leaves):
    """Memory and slots of a call on the current stream, before anything is timed or captured."""
    for _ in range(3):
        oal_b200.run_prepared_grouped_hd_block_gemm(prepared, *leaves)
    torch.cuda.current_stream().synchronize()


def test_a_stalled_call_keeps_its_status_word_and_delays_no_other_stream():
    """A training call behind half a second of other work, then more inference calls on another stream than there are
    slots: they finish first, and the stalled call's error is still reported."""
    from oal_b200 import hd_block_gemm_autograd as hd

    q, k, v, groups = _inputs(64, 4)
    bad = torch.full((4, 15), float("nan"), device="cuda").requires_grad_()
    good = torch.full((4, 15), 0.5, device="cuda")
    train = oal_b200.prepare_grouped_hd_block_gemm(q, k, v, groups, bad, precision="bf16_tensorcore")
    infer = oal_b200.prepare_grouped_hd_block_gemm(q, k, v, groups, good, precision="bf16_tensorcore")
    stalled, other = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(other):
        _warm(infer, q, k, v, good)
    torch.cuda.synchronize()
    with torch.cuda.stream(stalled):
        torch.cuda._sleep(2 * SLEEP)
        oal_b200.run_prepared_grouped_hd_block_gemm(train, q, k, v, bad)
        end = stalled.record_event()
    with torch.cuda.stream(other):
        for _ in range(1100):
            oal_b200.run_prepared_grouped_hd_block_gemm(infer, q, k, v, good)
            assert not end.query()
    with pytest.raises(RuntimeError, match=ERROR):
        hd.check_pending_status(block=True)
    assert end.query()
    for _ in range(5000):      # and the slots do not run out
        oal_b200.run_prepared_grouped_hd_block_gemm(infer, q, k, v, good)


def test_a_long_inference_call_waits_for_its_own_stream_only():
    q, k, v, groups = _inputs(64, 4)
    factor = torch.full((4, 15), 0.5, device="cuda")
    prepared = oal_b200.prepare_grouped_hd_block_gemm(q, k, v, groups, factor, precision="bf16_tensorcore")
    own, other = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(own):
        _warm(prepared, q, k, v, factor)
    torch.cuda.synchronize()
    with torch.cuda.stream(other):
        torch.cuda._sleep(2 * SLEEP)
        end = other.record_event()
    with torch.cuda.stream(own):
        torch.cuda._sleep(SLEEP // 5)
        oal_b200.run_prepared_grouped_hd_block_gemm(prepared, q, k, v, factor)
    assert not end.query()


def test_a_long_inference_call_beside_a_capture():
    """One thread records a graph while another waits for a call of 100 ms: both come through."""
    import threading

    q, k, v, groups = _inputs(64, 4)
    factor = torch.full((4, 15), 0.5, device="cuda")
    prepared = oal_b200.prepare_grouped_hd_block_gemm(q, k, v, groups, factor, precision="bf16_tensorcore")
    want = oal_b200.run_prepared_grouped_hd_block_gemm(prepared, q, k, v, factor)[0]
    stream, started, got = torch.cuda.Stream(), threading.Event(), []

    def wait_for_a_call():
        with torch.cuda.stream(stream):
            torch.cuda._sleep(SLEEP // 5)
            started.set()
            got.append(oal_b200.run_prepared_grouped_hd_block_gemm(prepared, q, k, v, factor)[0])

    with torch.cuda.stream(stream):
        _warm(prepared, q, k, v, factor)
    x = torch.zeros(8, device="cuda")
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    thread = threading.Thread(target=wait_for_a_call)
    with torch.cuda.graph(graph, capture_error_mode="thread_local"):      # other threads may allocate
        thread.start()
        started.wait()
        thread.join()
        x += 1
    graph.replay()
    torch.cuda.synchronize()
    assert x.eq(1).all() and torch.equal(got[0], want)


def _ticks(run):
    """The longest pause of another Python thread while ``run()`` is under way."""
    import threading
    import time

    stop, pauses = threading.Event(), [0.0]

    def tick():
        last = time.perf_counter()
        while not stop.is_set():
            time.sleep(0.001)
            now = time.perf_counter()
            pauses.append(now - last)
            last = now

    thread = threading.Thread(target=tick)
    thread.start()
    try:
        run()
    finally:
        stop.set()
        thread.join()
    return max(pauses)


def test_waiting_leaves_other_python_threads_running():
    """A full queue of unfinished training calls, an inference call and group ids that are not there yet: each waits
    for half a second or more of device work, without the interpreter's lock."""
    from oal_b200 import hd_block_gemm_autograd as hd

    q, k, v, groups = _inputs(64, 4)
    factor = torch.full((4, 15), 0.5, device="cuda")
    trained = factor.clone().requires_grad_()
    train = oal_b200.prepare_grouped_hd_block_gemm(q, k, v, groups, trained, precision="bf16_tensorcore")
    infer = oal_b200.prepare_grouped_hd_block_gemm(q, k, v, groups, factor, precision="bf16_tensorcore")
    stream = torch.cuda.Stream()

    def full_queue():
        torch.cuda._sleep(2 * SLEEP)
        for _ in range(260):
            oal_b200.run_prepared_grouped_hd_block_gemm(train, q, k, v, trained)

    def inference():
        torch.cuda._sleep(2 * SLEEP)
        oal_b200.run_prepared_grouped_hd_block_gemm(infer, q, k, v, factor)

    def late_ids():
        torch.cuda._sleep(2 * SLEEP)
        oal_b200.prepare_grouped_hd_block_gemm(q, k, v, groups + 0, factor, precision="bf16_tensorcore")

    with torch.cuda.stream(stream):
        _warm(train, q, k, v, trained)
        _warm(infer, q, k, v, factor)
        for run in (full_queue, inference, late_ids):
            assert _ticks(run) < 0.4, run.__name__
            torch.cuda.synchronize()
    hd.check_pending_status(block=True)


def test_one_preparation_from_two_threads_on_two_streams():
    import threading

    from oal_b200 import hd_block_gemm_autograd as hd

    q, k, v, groups = _inputs(300, 8)
    factor = torch.full((4, 45), 0.5, device="cuda")
    leaves = [t.clone().requires_grad_() for t in (q, k, v, factor)]
    prepared = oal_b200.prepare_grouped_hd_block_gemm(*leaves[:3], groups, leaves[3], precision="bf16_tensorcore")

    def step(scale):
        own = [(t * scale).detach().requires_grad_() for t in (q, k, v, factor)]
        out = oal_b200.run_prepared_grouped_hd_block_gemm(prepared, *own)[0]
        out.backward(torch.ones_like(out))
        return [out.detach(), *(t.grad for t in own)]

    want = {scale: step(scale) for scale in (1.0, 0.5)}
    torch.cuda.synchronize()
    got, errors = {1.0: [], 0.5: []}, []

    def work(scale):
        try:
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                for _ in range(50):
                    got[scale].append(step(scale))
            stream.synchronize()
        except Exception as exc:
            errors.append(exc)

    threads = [threading.Thread(target=work, args=(scale,)) for scale in got]
    for thread in threads:
        thread.start()
    for thread in threads:
        thread.join()
    hd.check_pending_status(block=True)
    assert not errors
    for scale, passes in got.items():
        for one in passes:
            for x, y in zip(one, want[scale]):
                assert torch.equal(x, y)
