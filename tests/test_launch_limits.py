"""Systems whose atoms fill a CTA's shared memory to the last bytes: the launch picker takes the
larger cluster exactly where the smaller one no longer fits beside the chain kernel's static part, so
every size in a range around that limit builds and runs.  Energies of the moved configuration against
its full recomputation, 1e-9 relative."""
import numpy as np
import pytest

from yamc_b200 import _lib, api, rng as grng, systems

pytestmark = pytest.mark.gpu


def _water(n, directory, kmax=10):
    box = (n / 0.015) ** (1 / 3)
    rc = min(9.0, 0.48 * box)
    spec = systems.SystemSpec("water", n, 0, 0, box, 3.0 / rc, rc, kmax)
    f = systems.write_system(spec, directory, seed=3)
    return api.load_inputs(f["parameters"], f["composition"], f["moltab"])


# one atom more is 40 bytes and a block of 32 atoms another 32, so the waters of the range step over
# the limit in parts of 120 bytes
@pytest.mark.parametrize("cluster,waters", [(1, range(1660, 1700)), (2, range(3330, 3390, 2))])
def test_every_size_around_the_shared_memory_limit_runs(tmp_path, cluster, waters):
    seen = set()
    moves = 6
    stream = grng.gfortran_stream(5, 60 * moves)
    for n in waters:
        b = api.Batch([_water(n, str(tmp_path / str(n)))])
        _, _, done, st, s = b.run([stream], moves)
        assert s == 0 and st[0] == 0 and done[0] == moves, n
        view = b.replica(0)
        assert np.all(np.abs(view.energies() - view.full_sums()) <= 1e-9 * np.maximum(np.abs(view.full_sums()), 1.0)), n
        seen.add(b.launch["cluster_blocks"])
        b.close()
    assert seen == {cluster, cluster + 1}


@pytest.mark.parametrize("kmax", [108, 110, 112, 127])  # phase tables of 46, 47 and 48 KB, and the largest
def test_per_move_calls_at_large_kmax(tmp_path, kmax):
    """The per-move pass's tables beside its static shared memory, around the 48 KB that need no leave:
    its energy change against that of the full sums, 1e-10 of the energies' scale."""
    inp = _water(12, str(tmp_path), kmax)
    eng = api.Engine(inp)
    e0 = eng.energies()
    eng.move_old(5)
    a, b = inp.first_atom[4] - 1, inp.last_atom[4]
    new = [v[a:b] + 0.004 for v in (inp.x, inp.y, inp.z)]
    du, overlap, _, _ = eng.move_eval(5, *new)
    assert not overlap
    eng.move_commit(True)
    assert np.all(np.abs(eng.energies() - eng.full_sums()) <= 1e-10 * np.abs(e0).max())
    assert abs(du[1] - (eng.energies()[6] - e0[6])) <= 1e-10 * np.abs(e0).max()


def test_a_refused_call_leaves_no_error_behind(tmp_path):
    """The runtime keeps the last error of a call until it is asked for: the calls after one that was
    refused must not report it."""
    inp = _water(12, str(tmp_path), 6)
    ok = api.Engine(inp)
    for _ in range(2):
        with pytest.raises(_lib.YamcError):
            api.Engine(inp, device=999)
        assert np.array_equal(ok.set_positions(inp.x, inp.y, inp.z), ok.full_sums())
        api.Engine(inp).close()
