"""The warp-drive right-hand side and projection on both sides of the radius beyond which its profile is exactly zero in
each precision, and a batch of every family whose launches run side by side, traced repeatedly on several streams.

Tolerance: where tanh rounds to 1 the profile and its gradient are zeros in the full form too, so the device metric equals
the oracle's to FP64 rounding (1e-13) on both sides of the edge; the batch equals its frames traced apart bit for bit."""
import numpy as np
import pytest

from sirius_b200 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sigma,R", [(8.0, 1.0), (2.0, 3.0), (30.0, 0.5)])
def test_profile_edge(engine, oracle, sigma, R):
    m = abi.make_metric(family=abi.ALCUBIERRE, vs=1.5, sigma=sigma, R=R)
    pts = []
    for t in (9.0, 9.3, 9.39, 9.41, 9.6, 19.0, 19.4, 19.49, 19.51, 19.8, 40.0):
        r = R + t / sigma
        for u in ((1, 0, 0), (0.6, 0.64, 0.48), (0, 0, -1)):
            pts.append([0.0, r * u[0], r * u[1], r * u[2]])
    g0, dg0 = oracle.metric_evaluate(m, np.array(pts))
    g, dg = engine.metric_evaluate(m, np.array(pts), abi.PRECISION_FP64)
    np.testing.assert_allclose(g, g0, rtol=0, atol=1e-13)
    np.testing.assert_allclose(dg, dg0, rtol=0, atol=1e-12 * sigma)
    gf, _ = engine.metric_evaluate(m, np.array(pts), abi.PRECISION_MIXED)
    np.testing.assert_allclose(gf, g0, rtol=0, atol=2e-6)


def test_side_by_side_batch_on_streams(engine):
    import torch
    frames, n = [], 0
    for i, (m, side) in enumerate([(abi.make_metric(a=0.9), 40), (abi.make_metric(family=abi.MORRIS_THORNE), 24),
                                   (abi.make_metric(family=abi.ALCUBIERRE), 17), (abi.make_metric(a=0.5, Lambda=1e-5), 9)]):
        frames.append(abi.make_frame(m, abi.make_camera(r=30.0, theta_deg=70.0, width=side, height=side + i), 0.0, 20.0,
                                     ray_offset=n))
        n += side * (side + i)
    engine.configure(abi.default_config(abs_tolerance=1e-7, rel_tolerance=1e-7, precision=abi.PRECISION_MIXED))
    size = abi.result_dtype().itemsize
    apart = b"".join(engine.trace_frames([abi.make_frame(f.metric, f.camera, 0.0, 20.0)])[0].tobytes() for f in frames)
    arr = (abi.Frame * len(frames))(*frames)
    d_frames = torch.from_numpy(np.frombuffer(bytes(arr), dtype=np.uint8).copy()).cuda()
    streams = [torch.cuda.Stream() for _ in range(2)]
    for k in range(6):
        s = streams[k % 2]
        out = torch.zeros(n * size, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        with torch.cuda.stream(s):
            engine.trace_frames_device(d_frames.data_ptr(), len(frames), n, out.data_ptr(), None, None, s.cuda_stream)
            host = out.cpu().numpy()  # ordered after the trace on its stream alone
        assert host.tobytes() == apart, k
