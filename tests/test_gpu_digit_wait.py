"""A digit product whose copy producer waits on a barrier that nothing arrives
on: L, dL and solve report it, and the context works on."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N", [(150, 9), (300, 40)])
def test_wait_runs_out(built, M, N):
    import pqdts_gb300 as pq
    from pqdts_gb300 import synth

    inst = synth.make_instance(M=M, N=N, D=2 * M, xmax=0.9 * M, eta=0.85, shots=10**6, gamma=1e-4, eps=1e-6, seed=3)
    rng = np.random.default_rng(2)
    X = rng.random((M, N)) + 0.1
    X = np.asfortranarray(X / X.sum(1, keepdims=True))

    def solver():
        s = pq.Solver(0)
        s.set_option("autotune", 0)
        s.set_instance(inst, pq.MIXED)
        assert s.get_option("sched.dg_fwd") == 1 and s.get_option("sched.dg_trans") == 1
        s.set_x(X)
        return s

    with solver() as s:
        L, G, H = s.L(), s.dL(), s.BF32(X)
    with solver() as s:
        s.set_option("tc_wait_ms", 5)
        s.set_option("tc_wait_probe", 1)
        for call in (s.L, s.dL, lambda: s.BF32(X), lambda: s.solve(mode=2, maxiter=1, eps=1e-6)):
            with pytest.raises(pq.PqdtsError, match=r"\(-2\).*barrier wait timed out"):
                call()
        s.set_option("tc_wait_probe", 0)
        s.set_option("tc_wait_ms", 2000)
        s.set_space(True, None)
        s.set_x(X)
        assert s.L() == L
        assert np.array_equal(s.dL(), G) and np.array_equal(s.BF32(X), H)
