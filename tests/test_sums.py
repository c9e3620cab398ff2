"""The whole-configuration sums over spatial tiles, at sizes around their edges (tiles of 32 atoms,
cell grids of 1 to 8 per axis) and with molecules outside the unit box, where the reference's single
conditional wrap and the nearest image differ: the tiles must hand over every pair that the wrap puts
inside the cutoff.  Real space against a direct numpy sum of all pairs, 1e-11 of the sum of magnitudes
(about 1e5 terms of FP64 rounding); forces against its gradient by the same formula; k space against
the unshifted configuration (whole-box shifts change no phase beyond rounding, 1e-11).  RDF counts
equal the oracle's."""
import math

import numpy as np
import pytest

import pyoracle
from yamc_b200 import api, systems

pytestmark = pytest.mark.gpu


def _erfc(x):
    x2, e2 = x * x, np.exp(-x * x)
    t = 1.0 / (1.0 + 0.3275911 * x)
    mid = t * (0.254829592 + t * (-0.284496736 + t * (1.421413741 + t * (-1.453152027 + t * 1.061405429)))) * e2
    low = 1.0 - 2.0 / 1.7724538509055 * x * (1.0 - x2 * (1 / 3 - x2 * (0.1 - x2 * (1 / 42 - x2 / 216))))
    far = (1.0 - 0.5 * (1.0 - 1.5 / x2) / x2) / (1.7724538509055 * x) * e2
    return np.where(x < 0.455, low, np.where(x > 3.0, far, mid))


def _real_space(inp, eng, x):
    """(uu_ew, uu_lj6, uu_lj12) and the sums of their magnitudes, every pair once."""
    p = eng.current_params()
    mol = np.repeat(np.arange(inp.nmol), inp.last_atom - inp.first_atom + 1)
    tot, mag = np.zeros(3), np.zeros(3)
    for i in range(len(x) - 1):
        d = x[i] - x[i + 1:]
        d = np.where(d > 0.5, d - 1.0, d)
        d = np.where(d < -0.5, d + 1.0, d)
        r2 = (d * d).sum(1)
        j = np.nonzero(r2 < p.rmax2)[0]
        r2, k = r2[j], j + i + 1
        r = np.sqrt(r2)
        a = p.alpha * r
        f = _erfc(a) - (mol[k] == mol[i])
        ew = p.xclb * inp.charge[i] * inp.charge[k] * f / r
        lj = (inp.sigma[i] > 1e-8) & (inp.sigma[k] > 1e-8)
        s6 = np.where(lj, ((inp.sigma[i] + inp.sigma[k]) / 2) ** 6 / r2 ** 3, 0.0)
        e4 = 4 * np.sqrt(inp.epsilon[i] * inp.epsilon[k]) * np.exp(-a * a)
        a2 = a * a
        c6 = 1 + a2 * (1 + a2 / 2)
        c12 = c6 + a2 ** 3 * (1 + a2 * (1 + a2 / 5) / 4) / 6
        for v, t in enumerate((ew, e4 * s6 * c6, e4 * s6 * s6 * c12)):
            tot[v] += t.sum()
            mag[v] += np.abs(t).sum()
    return tot, mag


@pytest.mark.parametrize("n_water,n_ion", [(10, 1), (11, 0), (85, 0), (171, 1), (700, 5)])
def test_real_space_tiles_with_molecules_outside_the_box(tmp_path, n_water, n_ion):
    box = ((n_water + 2 * n_ion) / 0.015) ** (1 / 3)
    rc = min(9.0, 0.48 * box)
    spec = systems.SystemSpec("odd", n_water, n_ion, n_ion, box, 3.2 / rc, rc, 5)
    files = systems.write_system(spec, str(tmp_path), seed=n_water)
    inp = api.load_inputs(files["parameters"], files["composition"], files["moltab"])
    eng = api.Engine(inp)
    base = eng.energies()
    f0 = eng.forces()[0]
    x = np.stack([inp.x, inp.y, inp.z], 1)
    tot, mag = _real_space(inp, eng, x)
    assert np.all(np.abs(base[3:6] - tot) <= 1e-11 * mag)
    r = np.random.default_rng(3)
    shift = r.integers(-1, 2, (inp.nmol, 3)) * (r.random((inp.nmol, 1)) < 0.3)
    y = x + np.repeat(shift, inp.last_atom - inp.first_atom + 1, axis=0)
    e = eng.set_positions(y[:, 0], y[:, 1], y[:, 2])
    tot, mag = _real_space(inp, eng, y)
    assert np.all(np.abs(e[3:6] - tot) <= 1e-11 * mag)
    assert np.all(np.abs(e[6:8] - base[6:8]) <= 1e-11 * np.abs(base[6:8]).max())
    eng.set_positions(*(np.ascontiguousarray(v) for v in x.T))
    assert np.abs(eng.forces()[0] - f0).max() <= 1e-12 * np.abs(f0).max()


@pytest.mark.parametrize("n_water,n_ion", [(2350, 3), (2355, 40)])
def test_force_rows_of_two_atoms_per_lane(tmp_path, n_water, n_ion):
    """Against the oracle's forces (erfc in place of erfc_Luc: 2e-4 of the force scale), and the same
    forces for molecules listed in another order (other lanes, blocks and halves of them)."""
    box = ((n_water + 2 * n_ion) / 0.0334) ** (1 / 3)
    spec = systems.SystemSpec("wide", n_water, n_ion, n_ion, box, 3.2 / 9.0, 9.0, 5)
    files = systems.write_system(spec, str(tmp_path), seed=n_water)
    inp = api.load_inputs(files["parameters"], files["composition"], files["moltab"])
    eng = api.Engine(inp)
    f, mf, _ = eng.forces()
    scale = math.sqrt((mf ** 2).sum(1).mean())
    o = pyoracle.Oracle(files)
    for imol in (1, 2, n_water // 2, n_water, n_water + 1, n_water + n_ion, n_water + 2 * n_ion):
        assert np.all(np.abs(o.move_old(imol)[0] - mf[imol - 1]) <= 2e-4 * scale)
    x = np.stack([inp.x, inp.y, inp.z], 1)
    perm = np.arange(len(x))
    perm[:3 * n_water] = perm[:3 * n_water].reshape(-1, 3)[::-1].ravel()
    perm[3 * n_water:3 * n_water + n_ion] = perm[3 * n_water:3 * n_water + n_ion][::-1]
    eng.set_positions(*(np.ascontiguousarray(v) for v in x[perm].T))
    assert np.abs(eng.forces()[0] - f[perm]).max() <= 1e-12 * np.abs(f).max()


@pytest.mark.parametrize("box", [31.0, 40.0])  # rmax above and below a third of the box
@pytest.mark.parametrize("m", [1023, 1024, 1057, 2001, 2399, 2400, 2433, 3599, 3600, 4001])
def test_rdf_tiles_count_as_all_pairs(m, box):
    r = np.random.default_rng(m)
    x, y, z = r.uniform(-0.5, 0.5, (3, m))
    x[::7] += 1.0   # outside the unit box: counted by the single conditional wrap
    z[::11] -= 1.0
    mol_type = np.where(np.arange(m) % 5 == 0, 2, 1).astype(np.int32)
    counts = np.array([(mol_type == 1).sum(), (mol_type == 2).sum()], dtype=np.int32)
    o = pyoracle.RDF(mol_type, counts, dr=0.1, rmax=12.0)
    o.add_frame(x, y, z, box)
    g = api.RDF(mol_type, counts, dr=0.1, rmax=12.0)
    g.add_frame(x, y, z, box)
    _, _, c, n = g.result()
    assert n == 1 and np.array_equal(c.ravel(), np.asarray(o.cnt4).ravel())
    assert c.sum() > 0 and math.isfinite(c.sum())


# remainders of a tile of 1, 31 and 0 above both thresholds of the tiles, and more tiles than one span of
# the near lists takes (1024)
@pytest.mark.parametrize("m,box", [(2401, 40.0), (2431, 40.0), (2432, 40.0), (3617, 31.0), (3647, 31.0), (3648, 31.0), (33001, 60.0)])
def test_rdf_tiles_count_as_all_pairs_at_their_edges(m, box):
    test_rdf_tiles_count_as_all_pairs(m, box)


def test_forces_over_more_than_one_span_of_tiles(nacl16k_files):
    """49,752 atoms, 1,555 tiles: against the oracle's forces as in the test above (2e-4 of the force
    scale), and the sum of all real-space and k-space pair forces, which is 0 but for rounding: 1e-9 of
    the sum of magnitudes (the sums of 1e5 terms of an atom are good to 1e-12 of theirs)."""
    inp = api.load_inputs(nacl16k_files["parameters"], nacl16k_files["composition"], nacl16k_files["moltab"])
    eng = api.Engine(inp)
    f, mf, _ = eng.forces()
    scale = math.sqrt((mf ** 2).sum(1).mean())
    o = pyoracle.Oracle(nacl16k_files)
    for imol in (1, 5461, 12000, 16384, 16385, 16684, 16984):
        assert np.all(np.abs(o.move_old(imol)[0] - mf[imol - 1]) <= 2e-4 * scale)
    assert np.all(np.abs(f.sum(0)) <= 1e-9 * np.abs(f).sum(0))
