"""Evaluations after a refused one: non-finite coordinates are refused, and once they are restored the forces,
energies and virials are those of the FP64 oracle again."""
import numpy as np
import pytest

from test_gpu_md import _melt_sim, _oracle_forces

pytestmark = pytest.mark.gpu


def _check(pd, ora, sim, q, box):
    pd.evaluate_forces_into_f(sim, energy=True)
    st = sim.state
    ref = _oracle_forces(pd, ora, sim, q, box)
    assert np.linalg.norm(st.forces() - ref["F"]) < 1e-5 * np.linalg.norm(ref["F"])   # the parity bound of the melt
    assert abs(st.potential_energy() - ref["Etot"]) < 1e-5 * abs(ref["Etot"])


@pytest.mark.parametrize("which", ["one", "all"])
@pytest.mark.parametrize("met_by", ["evaluation", "captured", "eager"])
def test_evaluation_after_non_finite_coordinates(pd, ora, cuda, which, met_by):
    sim, q, box = _melt_sim(pd, 4000, seed=11)
    st = sim.state
    pd.evaluate_forces_into_f(sim)
    st.step(2)
    st.synchronize()
    keep = [a.clone() for a in (st.x, st.y, st.z, st.vx, st.vy, st.vz, st.fx, st.fy, st.fz)]
    for _ in range(2):
        for a in (st.x, st.y, st.z):
            if which == "all":
                a.fill_(float("nan"))
            else:
                a[1234] = float("nan")
        if met_by == "evaluation":
            with pytest.raises(pd._native.NativeError, match="non-finite"):
                pd.evaluate_forces_into_f(sim)
        else:
            st.step(2, use_graph=met_by == "captured")
            st.synchronize()
        assert st.cluster.statistics()["error"] != 0
        for a, b in zip((st.x, st.y, st.z, st.vx, st.vy, st.vz, st.fx, st.fy, st.fz), keep):
            a.copy_(b)
        _check(pd, ora, sim, q, box)
    st.step(3)
    _check(pd, ora, sim, q, box)
