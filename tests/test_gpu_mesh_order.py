"""The mesh's own order of unordered charges: one chunk and one more, ragged counts, a flat box, gathers at moved
positions and of another count, against the FP64 oracle's mesh sum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,L", [(64, (14.0, 15.0, 16.0)), (65, (14.0, 15.0, 16.0)), (1501, (14.0, 15.0, 16.0)),
                                 (20011, (40.0, 44.0, 12.0)), (3000, (9.0, 9.0, 70.0))])
def test_unordered_charges(pd, ora, cuda, n, L):
    import torch
    rng = np.random.default_rng(n)
    mesh = tuple(int(2 * np.ceil(l / 2)) for l in L)
    R = (rng.random((n, 3)) * np.array(L) - np.array(L) / 2).astype(np.float32).astype(float)
    q = rng.standard_normal(n)
    q = (q - q.mean()).astype(np.float32).astype(float)
    spec = pd.ElectrostaticsSpec(coulomb_prefactor=1.7, real_cutoff=4.0, alpha=0.9, influence="spme", order=5, mesh=mesh,
                                 net_charge="background")
    s = pd.ElectrostaticsSolver(spec, L, q)
    t = [torch.tensor(np.ascontiguousarray(a), dtype=torch.float32, device="cuda") for a in (*R.T, q)]
    f = [torch.zeros(n, device="cuda") for _ in range(4)]
    s.transform(*t, energy=True)
    s.gather(*t, *f[:3], f[3], energy=True, set=True)
    torch.cuda.synchronize()
    ref = ora.mesh(R, q, L, mesh, 5, kind="spme", alpha=0.9, C=1.7, background=True)
    F = torch.stack(f[:3], 1).double().cpu().numpy()
    assert np.linalg.norm(F - ref["F"]) < 1e-5 * np.linalg.norm(ref["F"])   # the FP32 mesh bound
    assert np.linalg.norm(f[3].double().cpu().numpy() - ref["E"]) < 1e-5 * np.linalg.norm(ref["E"])
    # the same potential gathered with an explicit order, and at other positions, does not depend on the order
    perm = torch.tensor(rng.permutation(n), dtype=torch.int32, device="cuda")
    moved = [(a + 0.37).contiguous() for a in t[:3]] + [t[3]]
    out = []
    for order in (None, perm):
        g = [torch.zeros(n, device="cuda") for _ in range(3)]
        s.gather(*moved, *g, order=order, set=True)
        out.append(torch.stack(g))
    assert float((out[0] - out[1]).norm()) < 1e-6 * float(out[1].norm())
    half = n // 2   # fewer particles than the transform's
    g, h = ([torch.zeros(half, device="cuda") for _ in range(3)] for _ in range(2))
    m2 = [a[:half].contiguous() for a in moved]
    s.gather(*m2, *g, set=True)
    assert float((torch.stack(g) - out[1][:, :half]).norm()) < 1e-6 * float(out[1].norm())
    s.close()


def test_order_follows_the_stream(pd, cuda):
    """The own order belongs to the last transform that ran: captured ones that have not run yet, and replays between
    eager calls of other particle counts, leave every gather's particles complete."""
    import torch
    n, half, L = 3000, 1400, (14.0, 15.0, 16.0)
    rng = np.random.default_rng(8)
    R = rng.random((n, 3)) * np.array(L) - np.array(L) / 2
    q = rng.standard_normal(n)
    spec = pd.ElectrostaticsSpec(coulomb_prefactor=1.7, real_cutoff=4.0, alpha=0.9, influence="spme", order=5,
                                 mesh=(14, 16, 16), net_charge="background")
    s = pd.ElectrostaticsSolver(spec, L, q)
    t = [torch.tensor(np.ascontiguousarray(a), dtype=torch.float32, device="cuda") for a in (*R.T, q)]
    th = [a[:half].contiguous() for a in t]
    ident = torch.arange(n, dtype=torch.int32, device="cuda")

    def gather(x, order=None):
        g = [torch.zeros(x[0].numel(), device="cuda") for _ in range(3)]
        s.gather(*x, *g, order=order, set=True)
        return torch.stack(g)

    def agree(x):
        a, b = gather(x), gather(x, ident[:x[0].numel()].contiguous())
        # the same potential and stencils; only the FP32 brick offsets differ
        assert float((a - b).norm()) < 1e-6 * float(b.norm()) and float(b.norm()) > 0

    s.transform(*th)
    out = [torch.zeros(n, device="cuda") for _ in range(3)]
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):       # captured, not run
        s.transform(*t)
        s.gather(*t, *out, set=True)
    agree(t)                            # no order of n particles exists yet
    agree(th)
    for _ in range(2):
        graph.replay()                  # now the order holds n particles, though the last eager call had half
        torch.cuda.synchronize()
        b = gather(t, ident)
        assert float((torch.stack(out) - b).norm()) < 1e-6 * float(b.norm())
        agree(th)
        agree(t)
        s.transform(*th)
        agree(t)
        agree(th)
    s.close()


@pytest.mark.parametrize("order,alpha", [(5, 0.9), (6, 1.3), (8, 1.3)])
def test_sorted_charges_are_as_exact_as_unsorted(pd, ora, cuda, order, alpha):
    """Narrow splits leave the mesh sum exposed to the rounding of the charge grid.  Charges in a random order miss
    the spread's bricks and add in FP32; the mesh's own order adds in the bricks' fixed point."""
    import torch
    n, K = 12000, (60, 60, 60)
    Lx = (n / 0.0375) ** (1 / 3)
    rng = np.random.default_rng(3)
    R = (rng.random((n, 3)) * Lx - Lx / 2).astype(np.float32).astype(float)
    q = np.where(rng.random(n) < 0.5, 1.0, -1.0)
    q = (q - q.mean()).astype(np.float32).astype(float)
    spec = pd.ElectrostaticsSpec(coulomb_prefactor=1.7, real_cutoff=9.0, alpha=alpha, influence="spme", order=order,
                                 mesh=K, net_charge="background")
    s = pd.ElectrostaticsSolver(spec, (Lx,) * 3, q)
    t = [torch.tensor(np.ascontiguousarray(a), dtype=torch.float32, device="cuda") for a in (*R.T, q)]
    ref = ora.mesh(R, q, (Lx,) * 3, K, order, kind="spme", alpha=alpha, C=1.7, background=True)
    perm = torch.tensor(rng.permutation(n).astype(np.int32), device="cuda")
    err = []
    for o in (None, perm):
        f = [torch.zeros(n, device="cuda") for _ in range(3)]
        s.transform(*t, order=o)
        s.gather(*t, *f, order=perm, set=True)
        torch.cuda.synchronize()
        err.append(np.linalg.norm(torch.stack(f, 1).double().cpu().numpy() - ref["F"]))
    assert err[0] < 1.2 * err[1]   # the same rounding, other sums: within a fifth of each other
    s.close()
