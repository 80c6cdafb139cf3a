"""The quartet planner's kernels against plan_quartets (tensor operations, on the CPU): the
same quartets in the same class and precision part, every list ordered by decreasing primitive
quartets, the prefix of heavy quartets counted exactly."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _engine(name):
    from pychem_gb300 import workloads as W
    from pychem_gb300.engine import GpuEngine
    from pychem_gb300.ensemble import EnsembleEngine
    from pychem_gb300.molecule import Molecule
    if name == "ensemble":
        return EnsembleEngine([Molecule(c, "6-31G") for c in W.ensemble(13, seed=3)])
    if name == "atom":
        return GpuEngine(Molecule([["HE", 2.0, 0.0, 0.0, 0.0]], "STO-3G"))
    if name == "alkane":
        return GpuEngine(Molecule(W.alkane(3), "cc-pVDZ"))
    return GpuEngine(Molecule(W.water_cluster(nx=3, ny=2, nz=1), "6-31G"))


@pytest.mark.parametrize("thr,thr32", [(1e-8, 0.0), (1e-8, 1e-4), (1e-3, 1e-2), (0.0, 0.0), (10.0, 0.0), (1e30, 1e31)])
@pytest.mark.parametrize("name", ["atom", "water6", "alkane", "ensemble"])
def test_plan(name, thr, thr32):
    from pychem_gb300.engine import PARTS, plan_quartets
    eng = _engine(name)
    eng.one_electron()
    eng.schwarz()
    eng.threshold, eng.fp32_below = thr, thr32
    classes = eng.build_tasks()
    mol, nmol = eng._pair_molecules_host()
    pc = np.array([k[0] for k in eng.kinds])
    b, k = np.maximum(pc[:, None], pc[None, :]), np.minimum(pc[:, None], pc[None, :])
    plan, ket = plan_quartets(eng.Q.cpu(), torch.as_tensor(eng.pair_kind.astype(np.int64)), torch.as_tensor(mol), nmol,
                              torch.as_tensor(b * (b + 1) // 2 + k), thr, thr32,
                              kind_work=torch.as_tensor([k[1] for k in eng.kinds]))
    want = {}
    for cls, part, bra, off, qs, dg in plan:
        rows = want.setdefault((cls, part), [])
        for r in range(len(bra)):
            n = int(off[r + 1] - off[r])
            kets = ket[int(qs[r]):int(qs[r]) + n - int(dg[r])].tolist() + [int(bra[r])] * int(dg[r])
            rows += [(int(bra[r]), x) for x in kets]
    got = {(cls, part): t[0].view(-1, 2).cpu().numpy() for cls, rec in classes.items() for part, t in rec.items()}
    assert set(got) == set(want)
    npp = eng.h_npp
    for key, tasks in got.items():
        # plan_quartets may list a pair of one kind from its other side
        canon = lambda t: {(max(x), min(x)) if eng.pair_kind[x[0]] == eng.pair_kind[x[1]] else tuple(x) for x in t}
        assert len(canon(tasks.tolist())) == len(tasks) == len(want[key])
        assert canon(tasks.tolist()) == canon(want[key])
        work = npp[tasks[:, 0]] * npp[tasks[:, 1]]
        assert (np.diff(work) <= 0).all()
        assert eng.heavy[key] == tuple(np.count_nonzero(work >= k) for k in PARTS)
        assert classes[key[0]][key[1]][1] == len(tasks)
