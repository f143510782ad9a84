"""Captured steps across a change of the row capacity: the rows' stride and storage are the new ones, whatever
address the allocator returns."""
import numpy as np
import pytest

from test_gpu_learned import _ions, _params
from test_gpu_rows import _fluid

pytestmark = pytest.mark.gpu


# dense rows (the capacity is their stride), sparse rows, 2D
@pytest.mark.parametrize("dim,n,rho", [(3, 5000, 0.8), (3, 40000, 0.8), (3, 5000, 0.08), (2, 5000, 0.85)])
def test_captured_steps_follow_the_capacity(pd, ora, cuda, dim, n, rho):
    pos, box = _fluid(n, rho, 5 + n, dim)
    system = pd.ParticleSystem(pos, box, velocities=np.random.default_rng(2).normal(size=pos.shape))
    force = pd.LennardJones(epsilon=1.0, sigma=1.0, cutoff=2.5, neighborlist=pd.CellList(buffer=0.3, capacity=128))
    sim = pd.Simulation(system, pd.Integrator(dt=0.002, forces=[force]))
    st = sim.state
    st.step(3)
    for cap in (136, 128, 160, 128, 131):
        st.ell.resize(cap)
        st.engine.evaluate(stream=st.stream)   # eager: the rows are built with the new stride
        st.step(3)                              # captured
        st.synchronize()
        s = st.ell.status()
        assert s["error"] == 0 and s["cap"] == cap
        p = st.positions()
        p3 = p if dim == 3 else np.concatenate([p, np.zeros((n, 1))], 1)
        ref = ora.pairs_cells(p3, box if dim == 3 else (*box, 50.0), kind=1, sigma=1.0, eps=1.0, rc_lj=2.5)
        assert np.linalg.norm(st.forces() - ref["F"][:, :dim]) < 2e-5 * np.linalg.norm(ref["F"])   # the route's FP32 bound


def test_captured_learned_steps_follow_the_capacity(pd, cuda):
    n = 4000
    L = (n / 0.0375) ** (1.0 / 3.0)
    pos, q, typ, box = _ions(pd, n, L, 12)
    m = pd.synthetic.melt_masses(q)
    v = pd.synthetic.maxwell_boltzmann(m, 1200.0, seed=3, kB=pd.synthetic.KB_EV)
    system = pd.ParticleSystem(pos, box, types=["Na", "Cl"], typeids=typ, masses=m, charges=q, velocities=v)
    lj = pd.LennardJones(epsilon=0.01, sigma=2.8, cutoff=9.0, pairs="neighborlist",
                         neighborlist=pd.ClusterPairList(buffer=2.0, prune_buffer=0.6))
    el = pd.PME(coulomb_prefactor=pd.synthetic.COULOMB_EV_A, real_cutoff=9.0, real_space_tolerance=1e-5,
                mesh_spacing=2.0, order=4)
    st = pd.Simulation(system, pd.Integrator(dt=1.0 / pd.synthetic.TIME_UNIT_FS, forces=[lj, el])).state
    lc = pd.learned.LearnedCorrection(n, box, cap=128)
    lc.set_radial(np.linspace(0.01, -0.02, lc.nb))
    net = pd.learned.MLPNetwork(_params(pd, 1))
    st.engine.set_learned(lc, net)
    st.step(3)
    for cap in (160, 128, 144):
        st.synchronize()
        lc.resize(cap)
        st.engine.evaluate(stream=st.stream)
        st.step(2)
        F = st.forces()
        assert lc.status()["error"] == 0 and net.error() == 0
        st.engine.evaluate(stream=st.stream)   # the same positions, launched eagerly
        G = st.forces()
        # the same kernels on the same inputs; FP32 atomics reorder the sums
        assert np.linalg.norm(F - G) < 1e-5 * np.linalg.norm(G)
