"""Transform routes of the mesh engine at the edges of their size ranges, against the FP64 oracle's mesh sum
on the same mesh."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# planes in shared memory in place: smallest mesh, odd and unequal axes, radix 16 on every axis, a radix-1 factor;
# 736 threads on a plane; planes in two buffers (more items than threads); separate lines: large planes, odd rows and
# lines; cuFFT: 245 = 5 x 7 x 7, a prime factor 11
MESHES = [(5, 6, 7), (27, 25, 21), (16, 32, 256), (7, 120, 14), (120, 120, 6), (128, 128, 9), (160, 150, 7), (240, 256, 8),
          (225, 225, 6), (240, 225, 9), (225, 245, 6), (22, 26, 24)]


@pytest.mark.parametrize("influence", ["spme", "p3m_ik"])
@pytest.mark.parametrize("mesh", MESHES)
def test_transform_routes_match_the_oracle(pd, ora, cuda, mesh, influence):
    import torch
    L, C, rc, alpha, order = (14.0, 15.0, 16.0), 1.7, 4.0, 0.9, 5
    rng = np.random.default_rng(7)
    n = 200
    R = (rng.random((n, 3)) * np.array(L) - np.array(L) / 2).astype(np.float32).astype(float)
    q = rng.standard_normal(n)
    q = (q - q.mean()).astype(np.float32).astype(float)
    spec = pd.ElectrostaticsSpec(coulomb_prefactor=C, real_cutoff=rc, alpha=alpha, influence=influence, order=order,
                                 mesh=mesh, net_charge="background")
    s = pd.ElectrostaticsSolver(spec, L, q)
    x, y, z, qq = (torch.tensor(np.ascontiguousarray(a), dtype=torch.float32, device="cuda") for a in (*R.T, q))
    ref = ora.mesh(R, q, L, mesh, order, kind=influence, alpha=alpha, C=C, background=True)
    for energy in (True, False, True):   # the transform leaves the charge grid zero for the next
        f = [torch.zeros(n, device="cuda") for _ in range(4)]
        s.transform(x, y, z, qq, energy=energy)
        s.gather(x, y, z, qq, *f[:3], epot=f[3] if energy else None, energy=energy, set=True)
        torch.cuda.synchronize()
        F = torch.stack(f[:3], 1).double().cpu().numpy()
        # the parity bound of the FP32 mesh engine (test_gpu_mesh.py), relative to the largest of the forces
        # and of the rounding of the potential's gradient on very coarse meshes
        assert np.linalg.norm(F - ref["F"]) < 1e-5 * np.linalg.norm(ref["F"])
        if energy:
            assert abs(s.mesh_energy()[0] - ref["Emesh"]) < 1e-6 * abs(ref["Emesh"])
            assert abs(float(f[3].double().sum()) - ref["E"].sum()) < 1e-5 * np.abs(ref["E"]).sum()
    s.close()


@pytest.mark.parametrize("mesh", [(30, 32, 27), (128, 128, 24), (22, 32, 30)])
def test_batched_transform_routes(pd, ora, cuda, mesh):
    """Batched meshes: planes in place, planes in two buffers, cuFFT groups."""
    systems = pd.batch.melt_systems([600, 1000], seed=3)
    alpha, C, rc = pd.splits.alpha_from_tolerance(9.0, 1e-5), pd.synthetic.COULOMB_EV_A, 9.0
    b = pd.batch.BatchedReplicas(systems, skin=1.0, electrostatics=dict(alpha=alpha, C=C, rc=rc, order=5, mesh=mesh))
    for _ in range(2):
        b.evaluate(energy=True)
    for k, s in enumerate(systems):
        pos = np.stack([b.replica(k, t).cpu().numpy() for t in (b.x, b.y, b.z)], 1).astype(float)
        F = np.stack([b.replica(k, t).cpu().numpy() for t in (b.fx, b.fy, b.fz)], 1).astype(float)
        ref = ora.pme_total(pos, s["charges"], s["box"], C=C, alpha=alpha, rc=rc, K=mesh, P=5,
                            lj=dict(sigma=2.8, eps=0.01, rc=9.0))
        assert np.linalg.norm(F - ref["F"]) < 1e-5 * np.linalg.norm(ref["F"])
        assert abs(float(b.replica(k, b.epot).double().sum()) - ref["Etot"]) < 1e-5 * abs(ref["Etot"])
    b.close()


# z axes whose larger factor is odd (a half-empty last warp) and even, on planes and on separate lines
@pytest.mark.parametrize("influence", ["spme", "p3m_ik"])
@pytest.mark.parametrize("mesh", [(16, 18, 20), (14, 15, 42), (16, 15, 45), (12, 14, 54), (16, 16, 64), (15, 16, 72),
                                  (12, 12, 75), (10, 12, 81), (12, 10, 150), (8, 9, 225), (240, 256, 25)])
def test_energy_and_virial_of_every_warp_shape(pd, ora, cuda, mesh, influence):
    import torch
    L, C, alpha, order = (14.0, 15.0, 16.0), 1.7, 0.9, 5
    rng = np.random.default_rng(17)
    n = 300
    R = (rng.random((n, 3)) * np.array(L) - np.array(L) / 2).astype(np.float32).astype(float)
    q = rng.standard_normal(n)
    q = (q - q.mean()).astype(np.float32).astype(float)
    spec = pd.ElectrostaticsSpec(coulomb_prefactor=C, real_cutoff=4.0, alpha=alpha, influence=influence, order=order,
                                 mesh=mesh, net_charge="background")
    s = pd.ElectrostaticsSolver(spec, L, q)
    t = [torch.tensor(np.ascontiguousarray(a), dtype=torch.float32, device="cuda") for a in (*R.T, q)]
    ref = ora.mesh(R, q, L, mesh, order, kind=influence, alpha=alpha, C=C, background=True)
    for _ in range(3):
        f = [torch.zeros(n, device="cuda") for _ in range(4)]
        vg = torch.zeros(6, device="cuda")
        s.transform(*t, energy=True)
        s.gather(*t, *f[:3], epot=f[3], vglobal=vg, energy=True, set=influence != "p3m_ik")
        torch.cuda.synchronize()
        # FP64 sums over FP32 modes: the modes' rounding (a few 1e-7 of the energy) is all that is left
        assert abs(s.mesh_energy()[0] - ref["Emesh"]) < 1e-6 * abs(ref["Emesh"])
        assert np.max(np.abs(vg.double().cpu().numpy() - ref["W"])) < 2e-6 * abs(ref["Emesh"])
    s.close()
