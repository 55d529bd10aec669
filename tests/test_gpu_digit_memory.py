"""Device memory of the digit products' operands."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision, option", [("fp64", None), ("mixed", ("df_products", 1)), ("mixed", ("tensor_cores", 0))])
def test_given_back(built, small, precision, option):
    """A handle that is loaded with a problem that has no use for the operands
    gives them back, and takes them again for one that has."""
    import pqdts_gb300 as pq

    with pq.Solver(0) as s:
        s.set_option("autotune", 0)
        s.set_instance(small, pq.MIXED)
        held, L, G = s.get_option("sched.dg_bytes"), s.L(), s.dL()
        # F's 160 and F^T's 80 rows at least, of some chunks of 32 in eight slices
        assert held > (160 + 80) * 32 * 8 * 2
        if option:
            s.set_option(*option)
        s.set_instance(small, pq.MIXED if precision == "mixed" else pq.FP64)
        assert s.get_option("sched.dg_fwd") == 0 and s.get_option("sched.dg_bytes") == 0
        assert abs(s.L() - L) <= 1e-12 * L and abs(s.dL() - G).max() <= 1e-12 * abs(G).max()
        if option:
            s.set_option(option[0], -1)
        s.set_instance(small, pq.MIXED)
        assert s.get_option("sched.dg_bytes") == held
        assert s.L() == L and (s.dL() == G).all()


def test_limit(built, small):
    """Where the operands may not take their memory, double-FP32 it is, with
    the bits of df_products = 1; a limit that they meet leaves them in use."""
    import pqdts_gb300 as pq

    with pq.Solver(0) as s:
        s.set_option("autotune", 0)
        s.set_instance(small, pq.MIXED)
        held = s.get_option("sched.dg_bytes")
        s.set_option("digit_limit_mb", 0)
        s.set_instance(small, pq.MIXED)
        assert s.get_option("sched.dg_fwd") == 0 and s.get_option("sched.dg_bytes") == 0
        L, G = s.L(), s.dL()
        s.set_option("df_products", 1)
        s.set_instance(small, pq.MIXED)
        assert s.L() == L and (s.dL() == G).all()
        s.set_option("df_products", -1)
        s.set_option("digit_limit_mb", held // 2**20 + 1)
        s.set_instance(small, pq.MIXED)
        assert s.get_option("sched.dg_fwd") == 1 and s.get_option("sched.dg_bytes") == held
