"""The job server's planning kernel reads 128 jobs at a time and stops when the idle slots have run out: pools that run
out inside its first window of jobs, at its end, at the first job of the second, at the end of that, and not at all."""
import pytest

import pathtracer
from test_gpu_server import check_job, frame_renderers, make_server, resident, submit  # noqa: F401

pytestmark = pytest.mark.gpu


# a job has 4 pixels and one pass in flight, so it takes 4 slots: 257 jobs are two windows and one job
@pytest.mark.parametrize("pool", [4 * 100, 4 * 128, 4 * 128 + 1, 4 * 256, 4 * 300])
def test_slots_run_out_at_a_window_of_jobs(resident, frame_renderers, pool):  # noqa: F811
    srv, ids = make_server(resident, pool_size=pool, ring_passes=1, max_jobs=512, schedule=pathtracer.SCHEDULE_OLDEST_FIRST)
    try:
        jobs = [("cornell-all", 2, 2, 64, 6, True, 7 * k) for k in range(257)]
        jids = [submit(srv, ids, resident, job) for job in jobs]
        for jid, job in zip(jids, jobs):
            check_job(srv, jid, frame_renderers, resident, job)
    finally:
        srv.close()
