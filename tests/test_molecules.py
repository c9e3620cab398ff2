"""The chain kernel's k-space sweep over every shape of molecule, against the oracle.

A rigid 3-site molecule with charges on all sites and LJ on the first takes the sweep's short
form; every other shape (LJ on several sites, an uncharged LJ site, 1, 2 or 4 sites) the general
one.  Tolerances are those of the plain FP64 method: per-move dE within 1e-10 of max(|dE|, 1 kT),
identical decisions and stream cursors."""
import os

import numpy as np
import pytest

import pyoracle
from yamc_b200 import _lib, api, rng as grng, systems
from yamc_b200.formats import MolAtom, write_composition, write_mol, write_moltab, write_parameters

pytestmark = pytest.mark.gpu

O, H = (3.166, 0.1553), (0.0, 0.0)
SHAPES = {
    "water": [MolAtom("O", 0.0, 0.0, 0.0, *O, -0.8476, 16.0, 2.0), MolAtom("H", 1.0, 0.0, 0.0, *H, 0.4238, 0.0, 0.0),
              MolAtom("H", -0.33, 0.94, 0.0, *H, 0.4238, 0.0, 0.0)],
    "lj_on_all": [MolAtom("C", 0.0, 0.0, 0.0, 2.8, 0.05, 0.7, 12.0, 1.8), MolAtom("O", 1.16, 0.0, 0.0, *O, -0.35, 16.0, 2.0),
                  MolAtom("O", -1.16, 0.0, 0.0, *O, -0.35, 16.0, 2.0)],
    "neutral_site": [MolAtom("N", 0.55, 0.0, 0.0, 3.3, 0.07, -0.5, 14.0, 1.9), MolAtom("M", -0.55, 0.0, 0.0, 3.3, 0.07, 0.0, 14.0, 1.9),
                     MolAtom("Q", 0.0, 0.3, 0.0, *H, 0.2, 0.0, 0.0), MolAtom("Q", 0.0, -0.3, 0.2, *H, 0.3, 0.0, 0.0)],
    "pair": [MolAtom("A", 0.4, 0.0, 0.0, 2.584, 0.1, 0.5, 10.0, 1.8), MolAtom("B", -0.4, 0.0, 0.0, *H, -0.5, 4.0, 0.0)],
}


def _files(directory, xlambda):
    spec = systems.SystemSpec("shapes", 40, 0, 0, 17.0, 0.36, 8.0, 6, xlambda=xlambda)
    os.makedirs(directory, exist_ok=True)
    for name, atoms in SHAPES.items():
        write_mol(os.path.join(directory, name + ".mol"), atoms)
    comp, tab, prm = (os.path.join(directory, "system" + e) for e in (".composition", ".moltab", ".prm"))
    write_composition(comp, [(name + ".mol", 10) for name in SHAPES])
    write_moltab(tab, *systems.generate(spec, 4), 3, 3)
    write_parameters(prm, spec.params(0))
    return {"parameters": prm, "composition": comp, "moltab": tab, "dir": directory}


@pytest.mark.parametrize("xlambda", [0.0, 0.1])
@pytest.mark.parametrize("layout,cluster", [("registers", 2), ("registers", 3), ("streamed", 1), ("streamed", 2)])
def test_chain_of_every_molecule_shape(tmp_path, layout, cluster, xlambda):
    files = _files(str(tmp_path), xlambda)
    n = 400
    buf = grng.gfortran_stream(77, 60 * n)
    o = pyoracle.Oracle(files)
    olog, _, ocur = o.run_mc(buf, n)
    eng = api.Engine.from_files(files)
    eng.set_kspace_layout({"registers": _lib.YAMC_KSPACE_REGISTERS, "streamed": _lib.YAMC_KSPACE_STREAMED}[layout])
    eng.set_launch(cluster, 0)
    glog, _, gcur, done, st = eng.run_chain(buf, n)
    assert st == 0 and done == n and gcur == ocur
    assert len(np.unique(glog["imol"])) > 30  # molecules of every shape moved
    for k in ("imol", "flags", "cursor"):
        assert np.array_equal(glog[k], olog[k]), k
    for k in ("du_real", "du_k_coul", "du_k_lj", "du_ext"):
        assert np.all(np.abs(glog[k] - olog[k]) <= 1e-10 * np.maximum(np.abs(olog[k]), 1.0)), k
    assert np.all(np.abs(eng.energies() - o.energies()) <= 1e-9 * np.maximum(np.abs(o.energies()), 1.0))
