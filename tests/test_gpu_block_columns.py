"""Node-block GMRES replays recorded columns in long solves only: recording them costs
as much as ten columns, so a solve of a few columns launches its kernels."""
import pytest
import torch

from test_gpu_solver_threads import _Block

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q,columns,replays", [(0, 9, False), (1, 39, True)])
def test_short_solves_record_no_graph(cuda, q, columns, replays):
    job = _Block(1, cuda)
    job.solve(q)
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU, torch.profiler.ProfilerActivity.CUDA]) as prof:
        rc, it, x = job.solve(q)
    calls = [e.name for e in prof.events()]
    assert it == columns
    assert any("cudaLaunchKernel" in c for c in calls)
    assert any("cudaGraphLaunch" in c for c in calls) == replays
