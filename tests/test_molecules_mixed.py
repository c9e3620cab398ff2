"""The mixed form over the shapes of molecule that its k-space sweep does not take the short way (LJ on
several sites, an uncharged LJ site, four sites) beside rigid water, and its FP64 refresh of rho(k) over
the same, an uncharged site included.

Bars: those of the mixed form for a chain (dE within 1e-4 kT of the FP64 oracle's up to the first
decision that falls within that error); a refresh is FP64, so after one the k-space energies are those
of a full recomputation, 1e-11 of their magnitude (1e4 terms)."""
import os

import numpy as np
import pytest

import pyoracle
from test_molecules import SHAPES
from yamc_b200 import _lib, api, rng as grng, systems
from yamc_b200.formats import write_composition, write_mol, write_moltab, write_parameters

pytestmark = pytest.mark.gpu

NAMES = ("water", "lj_on_all", "neutral_site")  # three LJ types: what the mixed form takes


def _files(directory, xlambda, kmax):
    spec = systems.SystemSpec("shapes", 30, 0, 0, 17.0, 0.36, 8.0, kmax, xlambda=xlambda)
    os.makedirs(directory, exist_ok=True)
    for name in NAMES:
        write_mol(os.path.join(directory, name + ".mol"), SHAPES[name])
    comp, tab, prm = (os.path.join(directory, "system" + e) for e in (".composition", ".moltab", ".prm"))
    write_composition(comp, [(name + ".mol", 10) for name in NAMES])
    write_moltab(tab, *systems.generate(spec, 4), 3, 3)
    write_parameters(prm, spec.params(0))
    return {"parameters": prm, "composition": comp, "moltab": tab, "dir": directory}


def _engine(files, layout, cluster, threads):
    eng = api.Engine.from_files(files, precision=_lib.YAMC_MIXED)
    eng.set_kspace_layout({"registers": _lib.YAMC_KSPACE_REGISTERS, "streamed": _lib.YAMC_KSPACE_STREAMED}[layout])
    eng.set_launch(cluster, threads)
    return eng


@pytest.mark.parametrize("xlambda", [0.0, 0.1])
@pytest.mark.parametrize("layout,cluster,threads", [("registers", 2, 256), ("registers", 5, 128), ("streamed", 1, 256), ("streamed", 2, 384)])
def test_mixed_chain_of_every_molecule_shape(tmp_path, layout, cluster, threads, xlambda):
    files = _files(str(tmp_path), xlambda, 6)
    n = 400
    buf = grng.gfortran_stream(78, 60 * n)
    olog, _, _ = pyoracle.Oracle(files).run_mc(buf, n)
    glog, _, _, done, st = _engine(files, layout, cluster, threads).run_chain(buf, n)
    assert st == 0 and done == n
    same = (glog["flags"] == olog["flags"]) & (glog["cursor"] == olog["cursor"])
    k = n if same.all() else int(np.argmin(same))
    assert k >= 100 and len(np.unique(olog["imol"][:k])) > 20  # molecules of every shape moved
    du = ("du_real", "du_k_coul", "du_k_lj", "du_ext")
    assert np.abs(sum(glog[c][:k] for c in du) - sum(olog[c][:k] for c in du)).max() <= 1e-4


# entries per worker from less than one (idle warps) to several batches and a rest
@pytest.mark.parametrize("layout,cluster,threads,kmax", [
    ("registers", 2, 256, 6), ("registers", 9, 256, 12), ("streamed", 16, 384, 6), ("streamed", 1, 128, 6), ("streamed", 3, 256, 6),
    ("streamed", 1, 256, 12), ("streamed", 2, 384, 12), ("streamed", 3, 128, 12)])
def test_refresh_is_a_full_recomputation(tmp_path, layout, cluster, threads, kmax):
    eng = _engine(_files(str(tmp_path), 0.1, kmax), layout, cluster, threads)
    eng.set_refresh(1)
    buf = grng.gfortran_stream(79, 4000)
    cur, seen = 0, 0
    for _ in range(40):
        log, _, cur, done, st = eng.run_chain(buf, 1, cursor=cur)
        assert st == 0 and done == 1
        if log["flags"][0] & 1:
            seen += 1
            e, f = eng.energies(), eng.full_sums()
            assert np.all(np.abs(e[6:8] - f[6:8]) <= 1e-11 * np.maximum(np.abs(f[6:8]), 1.0))
    assert seen >= 5
