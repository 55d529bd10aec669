"""What set_problem derives on the device: Bdiag and the first maxr."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,D,width,gamma", [(2, 1, 1, 1, 0.0), (32, 3, 31, 7, 1e-3), (33, 70, 64, 33, 0.0),
                                               (65, 501, 129, 64, 1e-4), (300, 33, 1000, 40, 1e-3)])
def test_setup_bitwise(built, M, N, D, width, gamma):
    """Columns of F shorter, equal and longer than a block's steps of 32 rows,
    of uneven lengths, with zeros, tiny (2 f^2 subnormal) and large values:
    the oracle's bits."""
    import pqdts_gb300 as pq
    from oracle.oracle import Oracle
    from pqdts_gb300.synth import Instance

    rng = np.random.default_rng(M + N)
    lo = np.sort(rng.integers(0, M - width + 1, D)).astype(np.int64)
    val = rng.random(D * width) * 2.0 ** rng.integers(-20, 5, D * width)
    val[rng.random(val.size) < 0.05] = 0.0
    val[rng.random(val.size) < 0.05] = 1e-160
    P = rng.random((D, N))
    inst = Instance(M, N, D, gamma, 1e-6, lo, lo + width - 1, val, P / P.sum(1, keepdims=True))
    o = Oracle.from_instance(inst)
    with pq.Solver(0) as s:
        s.set_instance(inst)
        assert np.array_equal(s.Bdiag(), o.Bdiag())
        assert np.array_equal(s.maxr(), o.maxr())
