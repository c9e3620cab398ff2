"""A chain whose random stream ends at every position of its first moves: between a move's choice of
molecule and its proposal, inside the proposal, before the acceptance draw.  Every warp of every CTA
leaves the chain at the same move; the state is the one after the last whole move, and the rest of the
stream continues the run as if it had never stopped (the log of the uninterrupted run)."""
import numpy as np
import pytest

from yamc_b200 import _lib, api, rng as grng, systems

pytestmark = pytest.mark.gpu

MOVES = 4


@pytest.mark.parametrize("xlambda", [0.0, 0.1])
@pytest.mark.parametrize("layout,cluster,threads", [("registers", 1, 0), ("registers", 2, 128), ("streamed", 1, 384), ("streamed", 2, 0)])
def test_stream_end_at_every_position(tmp_path, layout, cluster, threads, xlambda):
    files = systems.write_system(systems.small_spec(xlambda=xlambda), str(tmp_path), seed=3)
    eng = api.Engine.from_files(files)
    eng.set_kspace_layout({"registers": _lib.YAMC_KSPACE_REGISTERS, "streamed": _lib.YAMC_KSPACE_STREAMED}[layout])
    eng.set_launch(cluster, threads)
    buf = grng.gfortran_stream(21, 400)
    start = eng.save_state(0)
    whole, _, end, done, st = eng.run_chain(buf, MOVES)
    assert st == 0 and done == MOVES
    bounds = [0] + [int(c) for c in whole["cursor"]]
    for n in range(0, end):
        eng.load_state(start)
        log, _, cur, done, st = eng.run_chain(buf[:n], MOVES)
        assert st == _lib.YAMC_ERNG_EXHAUSTED, n
        assert done < MOVES and cur == bounds[done] and cur <= n < bounds[done + 1], n
        rest, _, cur, more, st = eng.run_chain(buf, MOVES - done, cursor=cur)
        assert st == 0 and done + more == MOVES and cur == end, n
        both = np.concatenate([log, rest])
        assert all(np.array_equal(both[k], whole[k]) for k in ("imol", "flags", "cursor")), n
        for k in ("du_real", "du_k_coul", "du_k_lj", "du_ext"):
            assert np.all(np.abs(both[k] - whole[k]) <= 1e-10 * np.maximum(np.abs(whole[k]), 1.0)), (n, k)
