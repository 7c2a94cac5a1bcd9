"""The tuned cluster size of a batch belongs to the form of its solve."""
import pytest

from statfem_b200 import api
from tests.test_gpu_batch import make_batch, run_gpu

pytestmark = pytest.mark.gpu


def test_direct_and_iterative_entries(ctx, tmp_path):
    """The elimination and the iteration (a cap below 32 per line) are tuned
    and found separately."""
    api.autotune_clear()
    pb = make_batch([6, 12, 9], [4, 6, 5], 8)
    b, gm = run_gpu(ctx, pb, 1e-3)
    found = {}
    for cap in (50000, 300):
        b.set_solver(tol=1e-10, max_iter=cap)
        found[cap] = b.autotune()
        assert b.autotune() == found[cap] == b.launch_shape()[0]
        b.run()
        r = b.results()
        assert (r["status"] == 0).all() and r["iterations"].any() == (cap == 300)
    api.autotune_save(tmp_path / "t.txt")
    assert (tmp_path / "t.txt").read_text().count("batch:") == 2
    b.set_solver(tol=1e-10, max_iter=50000)
    assert b.autotune() == found[50000]
    b.close()
    gm.close()
