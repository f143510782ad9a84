"""The packed pair kernels over LJ kinds, Coulomb coefficient counts and CTA shapes: forces, energies and virials
against the FP64 pair sum, and the force-only pass against the energy pass."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lj", ["none", "uniform", "table"])
@pytest.mark.parametrize("alpha_rc,shape", [(0.0, (1, 1)), (1.5, (3, 4)), (3.12, (2, 2)), (4.4, (64, 1))])
def test_pair_tiles_match_the_oracle(pd, ora, cuda, lj, alpha_rc, shape):
    """alpha_rc: the split (more coefficients the larger it is; 0: no Coulomb term); shape: parts x warps."""
    import torch
    if lj == "none" and alpha_rc == 0.0:
        pytest.skip("no pair term")
    rng = np.random.default_rng(17)
    n, rc = 2213, 9.0
    Lb = (n / 0.0375) ** (1.0 / 3.0)
    box = (float(np.float32(Lb)),) * 3
    m = int(np.ceil(n ** (1 / 3) - 1e-9))
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pos = (g[rng.permutation(len(g))[:n]] + 0.5 + rng.uniform(-0.1, 0.1, (n, 3))) * (Lb / m) - Lb / 2
    pos = pos.astype(np.float32).astype(float)
    q = rng.choice([-1.0, 0.5, 1.0], n)
    kw, ref_kw = {}, {}
    if lj != "none":
        ref_kw.update(kind=1, sigma=2.8, eps=0.01, rc_lj=rc)
        if lj == "uniform":
            kw["lj"] = dict(table=pd.splits.lj_type_table(2.8, 0.01, rc))
        else:   # three types with one set of parameters: the table branch against the same sum
            one = np.full((3, 3), 1.0)
            kw["lj"] = dict(table=pd.splits.lj_type_table(2.8 * one, 0.01 * one, rc * one))
    else:
        ref_kw.update(kind=0)
    C = pd.synthetic.COULOMB_EV_A
    if alpha_rc > 0:
        alpha = alpha_rc / rc
        kw.update(coulomb=pd.splits.coulomb_polynomial(alpha, C, rc), selfc=0.0)
        ref_kw.update(q=q, C=C, alpha=alpha, rc_coul=rc)
    eng = pd.ClusterPairEngine(n, box, rmax=rc, skin=1.0, prune_buffer=0.3, **kw)
    eng.set_pair_shape(*shape)
    x, y, z, qq = (torch.tensor(np.ascontiguousarray(a), dtype=torch.float32, device="cuda") for a in (*pos.T, q))
    typ = torch.tensor(rng.integers(1, 4, n), dtype=torch.int32, device="cuda")
    out = []
    for energy in (True, False):
        f = [torch.zeros(n, device="cuda") for _ in range(4)]
        w = torch.zeros((n, 6), device="cuda")
        eng.compute(x, y, z, qq, typ, *f[:3], f[3], w, energy=energy)
        torch.cuda.synchronize()
        out.append((torch.stack(f[:3], 1).double().cpu().numpy(), f[3].double().cpu().numpy(),
                    w.double().cpu().numpy()))
    ref = ora.pairs_cells(pos, box, **ref_kw)
    (F, E, W), (F2, _, _) = out
    nF = np.linalg.norm(ref["F"])
    assert np.linalg.norm(F - ref["F"]) < 2e-5 * nF and np.linalg.norm(F2 - ref["F"]) < 2e-5 * nF
    assert np.linalg.norm(F - F2) < 2e-6 * nF
    assert np.linalg.norm(E - ref["E"]) < 2e-5 * np.linalg.norm(ref["E"])
    assert np.linalg.norm(W - ref["W"]) < 2e-5 * np.linalg.norm(ref["W"])
    eng.close()

