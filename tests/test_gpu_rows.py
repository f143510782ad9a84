"""Cell-order rows: row layouts, builds and force outputs at the sizes where their rules switch, against the
FP64 pair sums and the neighbour-row oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fluid(n, rho, seed, dim=3):
    """A jittered lattice of n particles at density rho, in random order."""
    rng = np.random.default_rng(seed)
    L = (n / rho) ** (1.0 / dim)
    m = int(np.ceil(n ** (1.0 / dim) - 1e-9))
    g = np.stack(np.meshgrid(*[np.arange(m)] * dim, indexing="ij"), -1).reshape(-1, dim)
    pos = (g[rng.permutation(len(g))[:n]] + 0.5 + rng.uniform(-0.12, 0.12, (n, dim))) * (L / m) - L / 2
    return pos.astype(np.float32).astype(float), (float(np.float32(L)),) * dim


# 3D, dense cells: a warp per row, the engine's lanes, forces by position; four and two warps per cell.
# Sparse cells: one thread per row, by particle and by position; 2D: the one-block and the tiled cell scan.
CASES = [(3, 1500, 0.8), (3, 17000, 0.8), (3, 33000, 0.8), (3, 9000, 0.08), (3, 40000, 0.08), (2, 9000, 0.85),
         (2, 60000, 0.85)]


@pytest.mark.parametrize("dim,n,rho", CASES)
def test_forces_and_rows(pd, ora, cuda, dim, n, rho):
    import torch
    pos, box = _fluid(n, rho, 5 + n, dim)
    rc, skin = 2.5, 0.3
    eng = pd.ELLEngine(n, box, dim=dim, model="lj", cutoff=rc, skin=skin, capacity=160)
    p3 = pos if dim == 3 else np.concatenate([pos, np.zeros((n, 1))], 1)
    b3 = box if dim == 3 else (*box, 50.0)
    ref = ora.pairs_cells(p3, b3, kind=1, sigma=1.0, eps=1.0, rc_lj=rc)
    x = [torch.tensor(np.ascontiguousarray(pos[:, d]), dtype=torch.float32, device="cuda") for d in range(dim)]
    x += [None] * (3 - dim)
    f = [torch.zeros(n, device="cuda") for _ in range(dim)] + [None] * (3 - dim)
    e, w = torch.zeros(n, device="cuda"), torch.zeros((n, 6 if dim == 3 else 3), device="cuda")
    eng.update(*x)
    eng.forces(*x, *f)
    torch.cuda.synchronize()
    F = torch.stack(f[:dim], 1).double().cpu().numpy()
    assert np.linalg.norm(F - ref["F"][:, :dim]) < 2e-5 * np.linalg.norm(ref["F"])   # the FP32 bound of the route
    eng.forces(*x, *f, epot=e, vir=w, energy=True)
    torch.cuda.synchronize()
    assert abs(float(e.double().sum()) - ref["E"].sum()) < 2e-5 * np.abs(ref["E"]).sum()
    W = ref["W"].sum(0) if dim == 3 else ref["W"].sum(0)[[0, 1, 3]]
    assert np.max(np.abs(w.double().sum(0).cpu().numpy() - W)) < 2e-5 * np.abs(W[:2]).sum()
    rows, counts = eng.rows_host()
    rl, sample = rc + skin, np.random.default_rng(1).integers(0, n, 300)
    L = np.array(b3)
    for i in sample:
        d = p3 - p3[i]
        d -= L * np.round(d / L)
        r = np.sqrt((d * d).sum(1))
        inner, outer = set(np.nonzero(r <= rl * (1 - 1e-5))[0]) - {i}, set(np.nonzero(r <= rl * (1 + 1e-5))[0]) - {i}
        got = set(rows[i].tolist())
        assert len(got) == counts[i] and inner <= got <= outer
    eng.close()


def test_exported_rows_follow_rebuilds(pd, cuda):
    """Rows read once stay current through later rebuilds, in eager updates and in captured steps."""
    import torch
    pos, box = _fluid(5000, 0.8, 3)
    system = pd.ParticleSystem(pos, box, velocities=np.random.default_rng(2).normal(size=pos.shape))
    force = pd.LennardJones(epsilon=1.0, sigma=1.0, cutoff=2.5, neighborlist=pd.CellList(buffer=0.3, capacity=160))
    sim = pd.Simulation(system, pd.Integrator(dt=0.005, forces=[force]))
    st = sim.state
    st.step(2)
    st.synchronize()
    st.ell.rows_host()
    st.ell.request(stream=st.stream)
    st.step(1)
    st.synchronize()
    rows, counts = st.ell.rows_host()
    p = st.positions()
    L = np.array(box)
    for i in range(0, 5000, 97):
        d = p - p[i]
        d -= L * np.round(d / L)
        r = np.sqrt((d * d).sum(1))
        got = set(rows[i].tolist())
        assert len(got) == counts[i]
        assert set(np.nonzero(r <= 2.8 * (1 - 1e-5))[0]) - {i} <= got <= set(np.nonzero(r <= 2.8 * (1 + 1e-5))[0]) - {i}


@pytest.mark.parametrize("nrep,n_hi", [(3, 1500), (12, 6000)])
def test_batch_outputs_match_single_systems(pd, cuda, nrep, n_hi):
    """Batched forces by particle (small batch) and by position (from 32 768 particles), and 8 captured steps."""
    import torch
    specs = pd.synthetic.replica_set(nrep, n_lo=1200 if nrep < 5 else 3000, n_hi=n_hi, seed=21)
    systems = pd.batch.make_systems(specs)
    b = pd.batch.BatchedReplicas(systems, skin=0.3, cap=160, lanes=1)
    b.evaluate()
    b.step(8, 0.004)
    b.synchronize()
    assert b.status()["error"] == 0 and (b.n >= 32768) == (nrep > 5)
    for k, s in enumerate(systems):
        t = [b.replica(k, a).clone() for a in (b.x, b.y, b.z)]
        kw = dict(model="lj", cutoff=2.5) if s["kind"] == "lj" else dict(model="wca")
        eng = pd.ELLEngine(s["n"], s["box"], skin=0.3, capacity=160, **kw)
        f = [torch.zeros(s["n"], device="cuda") for _ in range(3)]
        eng.update(*t)
        eng.forces(*t, *f)
        torch.cuda.synchronize()
        for a, c in zip((b.fx, b.fy, b.fz), f):
            assert float((b.replica(k, a) - c).norm()) < 1e-5 * float(torch.stack(f).norm())
        eng.close()


def _ell_forces(eng, x, n, dim=3, energy=False):
    import torch
    f = [torch.zeros(n, device="cuda") for _ in range(dim)] + [None] * (3 - dim)
    e, w = torch.zeros(n, device="cuda"), torch.zeros((n, 6 if dim == 3 else 3), device="cuda")
    eng.forces(*x, *f, epot=e if energy else None, vir=w if energy else None, energy=energy)
    torch.cuda.synchronize()
    return torch.stack(f[:dim], 1).double().cpu().numpy()


# dense rows, sparse rows, 2D; forces by particle and by position
@pytest.mark.parametrize("dim,n,rho", [(3, 1500, 0.8), (3, 33000, 0.8), (3, 9000, 0.08), (2, 9000, 0.85)])
@pytest.mark.parametrize("energy", [False, True])
def test_forces_at_uncentred_coordinates(pd, ora, cuda, dim, n, rho, energy):
    """Forces between updates take coordinates that have drifted over a face, or come as another image of the box."""
    import torch
    pos, box = _fluid(n, rho, 5 + n, dim)
    L = np.array(box)
    eng = pd.ELLEngine(n, box, dim=dim, model="lj", cutoff=2.5, skin=0.3, capacity=160)

    def dev(p):
        return [torch.tensor(np.ascontiguousarray(p[:, d]), dtype=torch.float32, device="cuda") for d in range(dim)] + \
               [None] * (3 - dim)

    eng.update(*dev(pos))
    rng = np.random.default_rng(4)
    moved = pos + 0.1 * rng.uniform(-1, 1, pos.shape) / np.sqrt(dim)      # within half the skin, not wrapped
    image = moved + L * (rng.random(pos.shape) < 0.2) * np.where(moved > 0, -1.0, 0.0)
    for p in (moved, image):
        p = p.astype(np.float32).astype(float)
        F = _ell_forces(eng, dev(p), n, dim, energy)
        p3 = p if dim == 3 else np.concatenate([p, np.zeros((n, 1))], 1)
        b3 = box if dim == 3 else (*box, 50.0)
        ref = ora.pairs_cells(p3 - np.array(b3) * np.round(p3 / np.array(b3)), b3, kind=1, sigma=1.0, eps=1.0, rc_lj=2.5)
        # FP32 coordinates up to a box from the centre: their rounding, through a force constant of about 1e3
        assert np.linalg.norm(F - ref["F"][:, :dim]) < 1e-4 * np.linalg.norm(ref["F"])
    eng.close()


@pytest.mark.parametrize("lanes", [1, 4])
@pytest.mark.parametrize("nrep,n_hi", [(3, 1500), (12, 6000)])
def test_batch_forces_at_uncentred_coordinates(pd, cuda, lanes, nrep, n_hi):
    """The same for the batched pass: another image of a particle, or one that has crossed a face, has the same pairs."""
    import torch
    specs = pd.synthetic.replica_set(nrep, n_lo=1200 if nrep < 5 else 3000, n_hi=n_hi, seed=21)
    b = pd.batch.BatchedReplicas(pd.batch.make_systems(specs), skin=0.3, cap=160, lanes=lanes)
    b.evaluate()
    b.synchronize()
    ref = torch.stack([b.fx, b.fy, b.fz]).double()
    rng = np.random.default_rng(3)
    img = []
    for d, a in enumerate((b.x, b.y, b.z)):
        t = a.clone()
        for k, s in enumerate(b.systems):
            v = b.replica(k, t)
            pick = torch.tensor(rng.random(s["n"]) < 0.2, device="cuda") & (v > 0)
            v -= pick * float(np.float32(s["box"][d]))
        img.append(t)
    f = [torch.zeros(b.n, device="cuda") for _ in range(3)]
    N = pd._native
    torch.cuda.synchronize()
    N.call("pd_batch_forces", b.handle, *[a.data_ptr() for a in img], *[a.data_ptr() for a in f], 0, 0, 0)
    torch.cuda.synchronize()
    # shifting a coordinate by a box rounds it to an ulp of the box, about 1e-6; force constants reach 1e3
    assert float((torch.stack(f).double() - ref).norm()) < 1e-4 * float(ref.norm())
    b.close()


@pytest.mark.parametrize("lanes", [0, 1, 4])
def test_non_finite_neighbour_leaves_the_rest(pd, ora, cuda, lanes):
    """A particle whose coordinate is not finite has no pairs: the other particles' forces stay finite."""
    import torch
    n = 1500
    pos, box = _fluid(n, 0.8, 12)
    eng = pd.ELLEngine(n, box, model="lj", cutoff=2.5, skin=0.3, capacity=160, lanes=lanes)
    x = [torch.tensor(np.ascontiguousarray(pos[:, d]), dtype=torch.float32, device="cuda") for d in range(3)]
    eng.update(*x)
    for bad in (float("nan"), float("inf")):
        y = [a.clone() for a in x]
        y[1][7] = bad
        for energy in (False, True):
            F = _ell_forces(eng, y, n, 3, energy)
            ref = ora.pairs_cells(np.delete(pos, 7, 0), box, kind=1, sigma=1.0, eps=1.0, rc_lj=2.5)
            assert np.linalg.norm(np.delete(F, 7, 0) - ref["F"]) < 2e-5 * np.linalg.norm(ref["F"])
    eng.close()


@pytest.mark.parametrize("lanes,charged", [(1, False), (4, False), (8, False), (1, True)])
def test_batch_non_finite_neighbour_leaves_the_rest(pd, cuda, lanes, charged):
    import torch
    if charged:
        el = dict(alpha=pd.splits.alpha_from_tolerance(9.0, 1e-5), C=pd.synthetic.COULOMB_EV_A, rc=9.0, order=5,
                  kind="spme", spacing=1.0)
        b = pd.batch.BatchedReplicas(pd.batch.melt_systems([1000, 1200], seed=3), skin=1.0, lanes=lanes, electrostatics=el)
    else:
        b = pd.batch.BatchedReplicas(pd.batch.make_systems(pd.synthetic.replica_set(3, n_lo=1200, n_hi=1500, seed=21)),
                                     skin=0.3, cap=160, lanes=lanes)
    b.evaluate()
    b.synchronize()
    for bad in (float("nan"), float("inf")):
        y = b.y.clone()
        y[700] = bad
        f = [torch.zeros(b.n, device="cuda") for _ in range(3)]
        torch.cuda.synchronize()
        pd._native.call("pd_batch_forces", b.handle, b.x.data_ptr(), y.data_ptr(), b.z.data_ptr(),
                        *[a.data_ptr() for a in f], 0, 0, 0)
        torch.cuda.synchronize()
        F = torch.stack(f)
        F[:, 700] = 0.0
        assert bool(torch.isfinite(F).all())
    b.close()


@pytest.mark.parametrize("dim,clump", [(3, 33), (3, 900), (2, 32), (2, 257)])
def test_rows_of_a_clump_in_a_sparse_box(pd, ora, cuda, dim, clump):
    """One crowded cell among sparse ones: its particles are in id order too, and every row is complete."""
    import torch
    n, L, rl = 6000, (60.0 if dim == 3 else 160.0), 2.8
    rng = np.random.default_rng(clump)
    pos = rng.uniform(-L / 2, L / 2, (n, dim))
    nc = int(L / rl)
    pos[rng.permutation(n)[:clump]] = (nc // 3 + 0.5) * (L / nc) - L / 2 + rng.uniform(-1.0, 1.0, (clump, dim))
    pos = pos.astype(np.float32).astype(float)
    eng = pd.ELLEngine(n, (L,) * dim, dim=dim, model="lj", cutoff=2.5, skin=0.3, capacity=1024)
    x = [torch.tensor(np.ascontiguousarray(pos[:, d]), dtype=torch.float32, device="cuda") for d in range(dim)]
    x += [None] * (3 - dim)
    eng.update(*x)
    assert eng.status()["error"] == 0
    rows, counts = eng.rows_host()
    p3 = pos if dim == 3 else np.concatenate([pos, np.zeros((n, 1))], 1)
    want = ora.neighbor_rows(p3, (L,) * 3, float(np.float32(2.5) + np.float32(0.3)), cap=1024)
    border = 0
    for i in range(n):
        got = sorted(rows[i].tolist())
        assert len(set(got)) == len(got) == counts[i]
        if got != want[i]:   # a pair whose distance is the list radius within an FP32 ulp
            for j in set(got) ^ set(want[i]):
                d = p3[i] - p3[j]
                r = np.linalg.norm(d - L * np.round(d / L))
                assert abs(r - rl) < 1e-5
                border += 1
    assert border < 20
    assert max(counts) >= clump // 2
    eng.request()   # id order inside a cell: a second build gives the same rows, entry by entry
    eng.update(*x)
    again, _ = eng.rows_host()
    assert all(np.array_equal(r, t) for r, t in zip(rows, again))
    eng.close()


@pytest.mark.parametrize("form", ["rows", "batch1", "batch4"])
def test_isolated_pairs_to_rounding(pd, cuda, form):
    """Every particle has one neighbour, so a force is one term.  With u = 2^-24: the differences and r^2 are within
    4 u, 1/r^2 (the refined approximation) adds 2 u, s2 u, so s6 is within 23 u, s12 within 47 u, and their products with
    1/r^2 and the difference within 58 u of the two terms' sizes."""
    import torch
    m, L = 1000, 60.0
    rng = np.random.default_rng(6)
    g = np.stack(np.meshgrid(*[np.arange(10)] * 3, indexing="ij"), -1).reshape(-1, 3) * 6.0 - 27.0
    d = rng.normal(size=(m, 3))
    d *= (np.linspace(0.72, 2.49, m) / np.linalg.norm(d, axis=1))[:, None]
    pos = np.stack([g + d / 2, g - d / 2], 1).reshape(-1, 3).astype(np.float32).astype(float)
    n = 2 * m
    x = [torch.tensor(np.ascontiguousarray(pos[:, k]), dtype=torch.float32, device="cuda") for k in range(3)]
    f = [torch.zeros(n, device="cuda") for _ in range(3)]
    e = torch.zeros(n, device="cuda")
    if form == "rows":
        eng = pd.ELLEngine(n, (L,) * 3, model="lj", cutoff=2.5, skin=0.3, capacity=8)
        eng.update(*x)
        eng.forces(*x, *f, epot=e, vir=torch.zeros((n, 6), device="cuda"), energy=True)
    else:
        eng = pd.batch.BatchedReplicas([dict(n=n, box=(L,) * 3, kind="lj", positions=pos, velocities=np.zeros((n, 3)),
                                             masses=1.0, eps=1.0, sigma=1.0, rc=2.5)], skin=0.3, cap=8,
                                       lanes=int(form[-1]))
        eng.evaluate(energy=True)
        eng.synchronize()
        f, e = [eng.fx, eng.fy, eng.fz], eng.epot
    torch.cuda.synchronize()
    F, E = torch.stack(f, 1).double().cpu().numpy(), e.double().cpu().numpy()
    r = pos[0::2] - pos[1::2]
    r2 = (r * r).sum(1)
    s6 = r2 ** -3
    u = 2.0 ** -24
    ref = (24.0 * (2.0 * s6 * s6 - s6) / r2)[:, None] * r
    size = 24.0 * (2.0 * s6 * s6 + s6) / np.sqrt(r2)
    assert np.all(np.abs(F[0::2] - ref) <= 58 * u * size[:, None]) and np.all(F[1::2] == -F[0::2])
    assert np.all(np.abs(E[0::2] - 2.0 * (s6 * s6 - s6)) <= 50 * u * 2.0 * (s6 * s6 + s6))
    eng.close()


@pytest.mark.parametrize("n,rho,asked,used", [(1500, 0.8, 0, 32), (1500, 0.8, 2, 2), (17000, 0.8, 0, 4), (9000, 0.08, 0, 1)])
def test_status_gives_the_lanes_in_use(pd, cuda, n, rho, asked, used):
    _, box = _fluid(n, rho, 3)
    eng = pd.ELLEngine(n, box, model="lj", cutoff=2.5, skin=0.3, capacity=160, lanes=asked)
    assert eng.status()["lanes"] == used
    eng.close()
