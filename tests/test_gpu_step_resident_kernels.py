"""The resident launches -- batches as bins in shared memory, scenes as a
thread-block cluster -- in a caller's buffers, where every call is one, against
the graph path of a context with a state of its own: re-sorts on every step, few
movers, unsorted starts, consecutive calls, both block sizes of the cluster, a
position that is no number."""
import numpy as np
import pytest

from demso_b200 import scenes
from helpers import same
from test_gpu_adopt import _sets, _view_np

pytestmark = pytest.mark.gpu

FIELDS = ("pos", "vel", "theta", "omega", "radius", "mass", "id")


def _t(a):
    import torch
    a = np.ascontiguousarray(a)
    return torch.from_numpy(a.view(np.int32).copy() if a.dtype == np.uint32 else a.copy())


def _context(parts, batch, flags):
    import demso_b200 as D
    flags |= D.CTX_PRESSURE | D.CTX_ACCEL
    if batch:
        return D.Batch([(p.sys, p.n) for p in parts], flags=flags)
    return D.Simulation(parts[0].sys, capacity=parts[0].n, flags=flags)


def _both(parts, batch, calls, shuffle=None, error=None):
    import torch
    import demso_b200 as D
    st = scenes.concat_specimens(parts) if batch else parts[0].state()
    if shuffle is not None:
        rng = np.random.default_rng(shuffle)
        at, order = 0, []
        for p in parts:
            order.append(at + rng.permutation(p.n))
            at += p.n
        order = np.concatenate(order)
        st = {k: (None if v is None else v[order]) for k, v in st.items()}
    n = st["pos"].shape[0]
    out = []
    for adopted in (True, False):
        sim = _context(parts, batch, D.CTX_RESIDENT | D.CTX_CALLER_STATE if adopted else 0)
        if adopted:
            first, second = _sets(st, False)
            sim.adopt_state(first, second, n)
        else:
            sim.set_state(*(_t(st[k]) for k in FIELDS))
        for k in calls:
            sim.step(k)
        torch.cuda.synchronize()
        if error is None:
            sim.check()
        else:
            with pytest.raises(D.DemError) as e:
                sim.check()
            assert e.value.code == error
        got = {k: v.numpy() for k, v in sim.get_state("cpu").items() if v is not None}
        if adopted:
            view = _view_np(sim.state_view())
            for k in FIELDS:
                assert np.array_equal(view[k][:n].view(np.uint32).reshape(-1),
                                      got[k].view(np.uint32).reshape(-1)), k
        out.append(got)
        sim.close()
    for k in FIELDS + ("loc", "pressure", "acc", "alpha"):
        assert same(out[0][k], out[1][k]), k


def _gases(counts, vel, omega=50.0, seed=90):
    vel = vel if isinstance(vel, tuple) else (vel,) * len(counts)
    return [scenes.agitated_gas(n=n, seed=seed + k, vel_std=v, omega_std=omega)
            for k, (n, v) in enumerate(zip(counts, vel))]


@pytest.mark.parametrize("calls", [(1,), (2,), (60,), (1, 9, 20, 17)])
def test_bins_of_mixed_specimens(calls):
    parts = [scenes.agitated_gas(n=700, seed=51),
             scenes.agitated_gas(n=300, seed=52, grid="ref", vel_std=1.0),
             scenes.settling_pile(side=24, box=0.06, seed=53, vel_std=0.3),
             scenes.agitated_gas(n=1200, seed=54, dt=1e-6),
             scenes.agitated_gas(n=90, seed=55, grid=(2, 2))]
    _both(parts, True, calls)


def test_bins_that_sort_on_every_step():
    _both(_gases((400, 900, 1500, 2600), 4.0, 500.0, 70), True, (80,))


def test_bins_with_few_movers():
    _both(_gases((2000, 3500, 1200, 800, 5000), (2.0, 1.0, 3.0, 0.5, 0.3)), True, (150,))


def test_bins_from_an_unsorted_state():
    _both(scenes.specimen_batch(num=40, seed=11, nmin=64, nmax=3000), True, (47,), shuffle=2)


def test_many_bins():
    _both(scenes.specimen_batch(num=512, seed=0, nmin=256, nmax=8192), True, (12,))


@pytest.mark.parametrize("n,vel,calls", [(3000, 1.0, (120,)), (1700, 4.0, (60,)),
                                         (7000, 0.5, (60,)), (8192, 0.3, (3, 20)),
                                         (2500, 0.8, (1, 12, 20))])
def test_cluster_launches(n, vel, calls):
    _both(_gases((n,), vel, 100.0, 7 + n), False, calls)


def test_cluster_pile_and_unsorted_start():
    _both([scenes.settling_pile()], False, (400,))
    _both(_gases((2500,), 0.8), False, (33,), shuffle=4)


@pytest.mark.parametrize("counts", [(1000, 500), (2200,)])
def test_a_position_that_is_no_number(counts):
    parts = _gases(counts, 0.5)
    parts[0].pos[10] = [np.nan, 0.01]
    _both(parts, len(counts) > 1, (6,), error=3)
