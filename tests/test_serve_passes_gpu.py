"""The server in passes of every size its dispatch tells apart, and with the
stage kernels throughout: each request as rendered alone."""
import numpy as np
import pytest

from cudaraytracer_b200.serve import RenderRequest, Server
from test_serve_gpu import mix, orbit, render_alone, resident  # noqa: F401 (resident is a fixture)

pytestmark = pytest.mark.gpu


def serve_and_compare(ctx, resident, reqs, monkeypatch=None, **config):
    srv = Server(ctx, **config)
    for sc in resident:
        srv.add_scene(sc)
    ids = [srv.submit(r) for r in reqs]
    srv.drain()
    got = [srv.result(rid, r.width, r.height) for rid, r in zip(ids, reqs)]
    srv.close()
    ctx.check_device_errors()
    if monkeypatch:
        monkeypatch.delenv("CRT_PATH_KERNEL")
    for r, g in zip(reqs, got):
        for x, y in zip(g, render_alone(resident[r.scene], r)):
            np.testing.assert_allclose(x, y, rtol=2e-5, atol=2e-6)


def test_served_small_passes_in_stages(crt_ctx, resident, monkeypatch):
    """The mixed requests of the server's test, in passes of 3,000 paths."""
    monkeypatch.setenv("CRT_PATH_KERNEL", "0")
    serve_and_compare(crt_ctx, resident, mix(resident), monkeypatch, paths_per_pass=3000, passes_in_flight=3)


@pytest.mark.parametrize("paths_per_pass", [300_000, 500_000, 1_000_000, 3_000_000])
@pytest.mark.parametrize("schedule", [Server.SHORTEST_FIRST, Server.ADMISSION_ORDER])
def test_served_passes_of_every_size(crt_ctx, resident, paths_per_pass, schedule):
    """Path kernel from the first bounce in both register budgets, from the
    second, and stages alone, with bounce limits on both sides of the
    hand-over."""
    cb, ico = resident
    reqs = [
        RenderRequest(0, 640, 512, 5, orbit(cb, 80, 10), seed=11),
        RenderRequest(1, 640, 480, 3, orbit(ico, 70, 200, 1.1), seed=12, max_bounces=1),
        RenderRequest(0, 301, 207, 4, orbit(cb, 100, 350, 0.9), seed=13, max_bounces=2),
        RenderRequest(1, 512, 512, 3, orbit(ico, 120, 30), seed=14, max_bounces=12, rr=0.6),
        RenderRequest(1, 173, 191, 5, orbit(ico, 45, 90, 0.8), seed=16, rr_start_bounce=2),
    ]
    serve_and_compare(crt_ctx, resident, reqs, paths_per_pass=paths_per_pass, passes_in_flight=2, schedule=schedule)
