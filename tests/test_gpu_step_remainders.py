"""Calls whose steps fill no pass of the step loop, at a size where the last ones
may be launches of their own: the state is that of calls of whole passes."""
import pytest

from demso_b200 import scenes
from helpers import gpu_run, same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1048576, 2200000])
def test_steps_that_fill_no_pass(n):
    sc = scenes.agitated_gas(n=n, seed=12, vel_std=0.2, pitch_factor=1.1, jitter=0.1)
    a = gpu_run(sc.sys, sc.state(), 68, chunks=[11, 7, 14, 3, 2, 1, 13, 17])
    b = gpu_run(sc.sys, sc.state(), 68, chunks=[12, 10, 10, 12, 12, 12])
    for k in ("pos", "vel", "theta", "omega", "id", "loc", "pressure", "acc", "alpha"):
        assert same(a[k], b[k]), k
