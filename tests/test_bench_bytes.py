"""The bench line's phase bytes where the Poisson solve runs as one launch."""
from tests.helpers import load_golden


def test_bench_poisson_bytes_of_a_solve_in_one_launch():
    """A solve that keeps its vectors on the chip moves no bytes per iteration:
    the operator and the vectors once per step."""
    import bench
    p, _ = load_golden("ve2d_oldroyd_log")
    nc, nnz = p.ncell, p.p_col.size
    for mixed in (False, True):
        few, _ = bench.phase_bytes(p, mixed, 2.0, 1.0 if mixed else 0.0, one_launch=True)
        many, _ = bench.phase_bytes(p, mixed, 20.0, 1.0 if mixed else 0.0, one_launch=True)
        assert few == many
        assert few["poisson_iter"] == 4 * (nc + 1) + nnz * (8 if mixed else 12) + 56 * nc + (36 * nc if mixed else 0)
        loop, _ = bench.phase_bytes(p, mixed, 2.0, 1.0 if mixed else 0.0)
        assert {k: v for k, v in loop.items() if k != "poisson_iter"} == {k: v for k, v in few.items() if k != "poisson_iter"}
