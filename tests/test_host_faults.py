"""The library's host code on a CUDA runtime of the tests' own (fake_cuda.py): what a call allocates and keeps, and what it
does when an allocation, a launch or a kernel's wait fails. No kernel runs: outputs are not looked at."""
import os
import shutil
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
import fake_cuda  # noqa: E402

from sirius_b200 import abi  # noqa: E402
from sirius_b200.engine import Engine, SiriusError, load_library  # noqa: E402

WEIGHTS = os.path.join(os.path.dirname(abi.__file__), "data", "surrogate_kerr.npy")
MLP, MLP_FLAG = "mlp_pair_kernel", 4  # the inference kernel and the place of its error flag among its arguments


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    return fake_cuda.link(str(tmp_path_factory.mktemp("fake")))


@pytest.fixture
def fake(library):
    f = fake_cuda.Fake(library)
    f.reset()
    yield f
    f.reset()


@pytest.fixture
def eng(library, fake):
    e = Engine(0, lib=load_library(library))
    yield e
    e.close()
    assert fake.device_bytes == 0 and fake.pinned == 0 and fake.streams == 0 and fake.events == 0


def weights():
    return np.load(WEIGHTS).astype(np.float32).ravel()


def infer(eng, n=300):
    x, y = np.zeros((n, 5), np.float32), np.zeros((n, 4), np.float32)
    eng.surrogate_infer(x.ctypes.data, n, y.ctypes.data)


def test_weights_take_no_page_locked_memory(eng, fake):
    eng.surrogate_load(weights())
    assert fake.pinned == 0
    fake.reset()
    infer(eng)
    assert fake.calls("cudaMemcpyAsync") == fake.calls("cudaMemsetAsync") == 0 and fake.launches(MLP) == 1


@pytest.mark.parametrize("watchdog,sync", [(50, 0), (200, 120)])
def test_a_wait_that_ran_out_is_reported_and_cleared(eng, fake, watchdog, sync):
    """A call that took long enough for a wait to run out, or whose bound is short, reads the kernel's flag."""
    eng.configure(abi.default_config(watchdog_ms=watchdog))
    eng.surrogate_load(weights())
    infer(eng)
    fake.hook(MLP, MLP_FLAG, 1)
    fake.sync_ms(sync)
    with pytest.raises(SiriusError) as e:
        infer(eng)
    assert e.value.code == abi.ERR_TIMEOUT
    fake.reset()
    fake.sync_ms(sync)
    infer(eng)  # flag and counter start over
    assert fake.calls("cudaMemsetAsync") == 1
    infer(eng)
    assert fake.calls("cudaMemsetAsync") == 1


def frame(w=32, h=32, **metric):
    cam = abi.make_camera(r=100.0, theta_deg=60.0, width=w, height=h, fov=30.0)
    return abi.make_frame(abi.make_metric(**(metric or {"a": 0.9})), cam, 0.0, 30.0)


def features(eng):
    x, gate = np.zeros((32 * 32, 5), np.float32), np.zeros(32 * 32, np.uint8)
    eng.surrogate_features([frame()], x.ctypes.data, gate.ctypes.data)


def test_features_report_a_wait_that_ran_out(eng, fake):
    """The gate rests on the network's coarse pass: its error is the call's."""
    eng.configure(abi.default_config(watchdog_ms=50))
    features(eng)  # without weights there is no coarse pass, and no error to read
    eng.surrogate_load(weights())
    features(eng)
    fake.hook(MLP, MLP_FLAG, 1)
    with pytest.raises(SiriusError) as e:
        features(eng)
    assert e.value.code == abi.ERR_TIMEOUT
    fake.reset()
    features(eng)


def render(eng):
    img, gate = np.zeros(32 * 32, np.float32), np.zeros(32 * 32, np.uint8)
    eng.render_surrogate_device([frame()], img.ctypes.data, None, gate.ctypes.data)


def failures(fake, name, call):
    """Have the 1st, 2nd, ... call of a runtime function within `call` fail, each in a call of its own; yields after each."""
    nth = 1
    while True:
        fake.reset()
        fake.fail(name, nth, fake_cuda.INVALID_VALUE)
        try:
            call()
        except SiriusError:
            yield nth
        else:
            break
        nth += 1
    assert nth > 1
    fake.reset()


@pytest.mark.parametrize("call,name", [(c, n) for c, names in (
    (render, "cudaLaunchKernel cudaEventRecord cudaMemcpyAsync cudaMemsetAsync cudaStreamWaitEvent cudaEventSynchronize "
             "cudaStreamSynchronize"),
    (features, "cudaLaunchKernel cudaMemcpyAsync cudaStreamSynchronize"),
    (infer, "cudaStreamSynchronize")) for n in names.split()])
def test_error_exits_leave_no_network_launch_in_flight(eng, fake, name, call):
    """A call that fails after it launched the network waits for what it has launched, and the next call starts the
    kernel's counter over."""
    eng.configure(abi.default_config(precision=abi.PRECISION_MIXED))
    eng.surrogate_load(weights())
    call(eng)
    seen = 0
    for _ in failures(fake, name, lambda: call(eng)):
        if fake.launches(MLP) == 0:
            continue
        seen += 1
        assert fake.pending == 0
        fake.reset()
        call(eng)
        assert fake.calls("cudaMemsetAsync") >= 1 and fake.pending == 0
    assert seen > 0


def batch():
    """Frames of two families: their launches run side by side, one of them on a stream of the library's own."""
    frames, n = [], 0
    for m in ({"a": 0.9}, {"family": abi.MORRIS_THORNE}, {"a": 0.5}):
        f = frame(16, 8, **m)
        f.ray_offset = n
        n += 16 * 8
        frames.append(f)
    return (abi.Frame * len(frames))(*frames), len(frames), n


@pytest.mark.parametrize("name", ["cudaLaunchKernel", "cudaEventRecord", "cudaStreamWaitEvent"])
def test_error_exits_of_a_batch_leave_no_side_launch_in_flight(eng, fake, name):
    """Whatever fails, a caller that waits for its own stream has waited for every launch."""
    import ctypes
    arr, k, n = batch()
    img = np.zeros(n, np.float32)

    def call():
        eng.trace_frames_device(ctypes.addressof(arr), k, n, None, img.ctypes.data, None, None)

    eng.configure(abi.default_config(precision=abi.PRECISION_MIXED))
    call()
    assert fake.launches("trace_kernel") == 2 and fake.pending_own > 0
    for _ in failures(fake, name, call):
        fake.wait()
        assert fake.pending_own == 0


def test_a_batch_makes_the_streams_and_events_it_uses(eng, fake):
    """One stream and one event for each launch after the first, and the event they wait for."""
    import ctypes
    arr, k, n = batch()
    img = np.zeros(n, np.float32)
    eng.configure(abi.default_config(precision=abi.PRECISION_MIXED))
    streams, events = fake.streams, fake.events
    eng.trace_frames_device(ctypes.addressof(arr), 1, 16 * 8, None, img.ctypes.data, None, None)
    assert (fake.streams, fake.events) == (streams, events)
    for _ in range(2):
        eng.trace_frames_device(ctypes.addressof(arr), k, n, None, img.ctypes.data, None, None)
        assert (fake.streams, fake.events) == (streams + 1, events + 2)
    big = frame(512, 512)  # traced in pieces into host memory
    eng.trace_frames([big])
    many = fake.streams, fake.events
    assert many[0] > streams + 1
    eng.trace_frames([big])
    eng.trace_frames_device(ctypes.addressof(arr), k, n, None, img.ctypes.data, None, None)
    assert (fake.streams, fake.events) == many


def training_set(n):
    return np.zeros((n, 5), np.float32), np.zeros((n, 4), np.float32), np.ones(n, np.float32)


def gradient(eng, n=256):
    x, t, w = training_set(n)
    return eng.train_gradient(x.ctypes.data, t.ctypes.data, w.ctypes.data, n)


def test_training_without_tensor_maps(library, tmp_path):
    """A driver that encodes no tensor maps: every operand goes through registers. (A copy of the library: it asks the
    driver once.)"""
    path = str(tmp_path / "libsirius_fake_no_maps.so")
    shutil.copy(library, path)
    fake = fake_cuda.Fake(path)
    fake.fail("cudaGetDriverEntryPoint", 1, fake_cuda.NOT_SUPPORTED)
    eng = Engine(0, lib=load_library(path))
    try:
        eng.train_init(weights(), abi.train_config(batch=256))
        fake.reset()
        gradient(eng)
        assert fake.launches("train_forward_kernel") == 1 and fake.launches("gemm_kernel") == 9
    finally:
        eng.close()


def test_training_rows_are_one_allocation(eng, fake):
    """A batch's 15 buffers: one allocation, released with the next larger batch."""
    fake.reset()
    eng.train_init(weights(), abi.train_config(batch=256))
    assert fake.calls("cudaMalloc") <= 8
    small = fake.device_bytes
    eng.train_init(weights(), abi.train_config(batch=512))
    grown = fake.device_bytes
    per_row = 2 * (16 + 16 + 8 * 256) + 4 * (4 * 256 + 4 + 1 + 4)
    assert abs((grown - small) - 256 * per_row) <= 15 * 1024
    fake.reset()
    eng.train_init(weights(), abi.train_config(batch=256))
    assert fake.calls("cudaMalloc") == 0 and fake.device_bytes == grown
    gradient(eng)


@pytest.mark.parametrize("first", [True, False])
def test_training_whose_memory_ran_out_is_refused_until_it_is_made(eng, fake, first):
    """An initialisation that ran out of memory leaves no state that a step, an evaluation or a gradient would run on."""
    if not first:
        eng.train_init(weights(), abi.train_config(batch=256))
        gradient(eng)
    nth = 0
    while True:
        nth += 1
        fake.reset()
        fake.fail("cudaMalloc", nth)
        try:
            eng.train_init(weights(), abi.train_config(batch=512 + 128 * nth))
        except SiriusError as e:
            assert e.code == abi.ERR_OUT_OF_MEMORY
        else:
            break
        fake.reset()
        x, t, w = (a.ctypes.data for a in training_set(2048))
        calls = [lambda: gradient(eng), lambda: eng.train_steps(x, t, w, 2048, 1),
                 lambda: eng.train_evaluate(x, t, w, 2048)]
        if first:
            calls.append(lambda: eng.train_params())
        else:
            eng.train_params()  # those of the initialisation before
        for call in calls:
            with pytest.raises(SiriusError) as r:
                call()
            assert r.value.code == abi.ERR_NOT_CONFIGURED
        assert fake.launches("") == 0
    assert nth == (9 if first else 2)
    gradient(eng)
    eng.train_params()


def test_an_error_is_reported_once(eng, fake):
    """A call that ran out of memory is answered by that call, not by the next one's launch check."""
    eng.surrogate_load(weights())
    fake.fail("cudaMalloc", 1)
    with pytest.raises(SiriusError) as r:
        render(eng)
    assert r.value.code == abi.ERR_OUT_OF_MEMORY
    infer(eng)
    render(eng)


@pytest.mark.parametrize("name,n", [("cudaMalloc", 1), ("cudaMalloc", 2), ("cudaMemsetAsync", 1),
                                    ("cudaFuncSetAttribute", 1), ("cudaMemcpyAsync", 1), ("cudaStreamSynchronize", 1)])
def test_weights_whose_load_failed_are_not_there(eng, fake, name, n):
    """A first load that failed half-way leaves the network unloaded, and can be repeated."""
    fake.reset()
    fake.fail(name, n)
    with pytest.raises(SiriusError):
        eng.surrogate_load(weights())
    for rows in (0, 300):
        with pytest.raises(SiriusError) as r:
            infer(eng, rows)
        assert r.value.code == abi.ERR_NOT_CONFIGURED
    features(eng)
    assert fake.launches(MLP) == 0
    eng.surrogate_load(weights())
    infer(eng, 0)
    infer(eng)
    assert fake.launches(MLP) == 1


def evaluate(eng, n):
    eng.metric_evaluate(abi.make_metric(a=0.5), np.ones((n, 4)))


def step(eng, n):
    eng.dp45_step(abi.make_metric(a=0.5), np.ones((n, 8)), np.ones(n))


def beams(eng, n):
    eng.trace_beams([frame(n, 1)])


@pytest.mark.parametrize("call,row", [(evaluate, 84 * 8), (step, 84), (beams, 32)])
def test_a_large_calls_workspace_is_given_back(eng, fake, call, row):
    """The calls on host buffers keep a small workspace from one call to the next, not a large one."""
    call(eng, 1000)
    before = fake.device_bytes
    fake.reset()
    call(eng, 1000)
    assert fake.calls("cudaMalloc") == 0 and fake.device_bytes == before
    large = (64 << 20) // row + 1000
    call(eng, large)
    assert fake.device_bytes <= before
    call(eng, 1000)
    assert fake.device_bytes <= before


def test_a_handle_asks_for_the_attributes_it_needs(library, fake):
    """A new handle does not query the whole property record; a device before compute capability 10 is refused."""
    lib = load_library(library)
    e = Engine(0, lib=lib)
    assert fake.calls("cudaGetDeviceProperties") == 0
    e.close()
    fake.major(9)
    with pytest.raises(SiriusError) as r:
        Engine(0, lib=lib)
    assert r.value.code == abi.ERR_UNSUPPORTED
    fake.major(10)
    for n in (1, 2):
        fake.fail("cudaDeviceGetAttribute", n, fake_cuda.INVALID_VALUE)
        with pytest.raises(SiriusError) as r:
            Engine(0, lib=lib)
        assert r.value.code == abi.ERR_CUDA


def test_waits_of_an_error_exit_leave_no_error_behind(eng, fake):
    """Where the wait of an error exit fails as well, the call's own error is reported and the next call runs."""
    import ctypes
    eng.configure(abi.default_config(precision=abi.PRECISION_MIXED))
    eng.surrogate_load(weights())
    render(eng)
    arr, k, n = batch()
    img = np.zeros(n, np.float32)

    def trace():
        eng.trace_frames_device(ctypes.addressof(arr), k, n, None, img.ctypes.data, None, None)

    trace()
    # (a trace waits once for its caller's stream before it launches)
    for call, nth, wait in ((render, 3, 1), (lambda e: trace(), 2, 2)):
        fake.reset()
        fake.fail("cudaStreamWaitEvent", nth, fake_cuda.INVALID_VALUE)
        fake.fail("cudaStreamSynchronize", wait, fake_cuda.NOT_SUPPORTED)
        with pytest.raises(SiriusError) as r:
            call(eng)
        assert "cudaStreamWaitEvent" in str(r.value) and fake.calls("cudaStreamSynchronize") >= wait
        infer(eng)
        render(eng)
        trace()
