"""DeviceProblem.kernel_launches against the launch sequence of one evaluation
(csrc/sv_loglik.cu, run_eval): three set-up kernels, the tables, the blocks, the
chunks' levels and their re-evaluation, four reductions."""
import pytest

CASES = [  # blocks in warps, in CTAs, d, precision, chunked, nu, estimated, kernels
    (500, 0, 4, "float64", True, 2.5, False, 3 + 3 + 2 + 4),   # fixed point, half, warp; levels, fix-up
    (500, 0, 4, "float64", False, 2.5, False, 3 + 3 + 4),
    (500, 0, 4, "float64", True, 0.5, False, 3 + 2 + 2 + 4),
    (500, 0, 13, "float64", True, 2.5, False, 3 + 2 + 2 + 4),
    (500, 0, 4, "float64", True, 1.3, False, 3 + 1 + 2 + 2 + 4),
    (500, 0, 4, "float64", True, None, True, 3 + 1 + 2 + 2 + 4),
    (500, 0, 4, "split", True, 2.5, False, 3 + 2 + 2 + 2 + 4),  # pre-pass, split; levels, fix-up; half, warp
    (500, 0, 4, "split_df", True, 1.3, False, 3 + 2 + 2 + 2 + 2 + 4),
    (31, 400, 4, "float64", True, 2.5, False, 3 + 3 + 1 + 3 + 4),
    (0, 400, 4, "float64", True, 2.5, False, 3 + 1 + 2 + 4)]


@pytest.mark.parametrize("warp,cta,d,precision,chunked,nu,est,kernels", CASES)
def test_count(warp, cta, d, precision, chunked, nu, est, kernels):
    from pyscaledvecchia_gb300.likelihood import DeviceProblem
    prob = DeviceProblem.__new__(DeviceProblem)
    prob.nblk, prob.nblk_warp, prob.d, prob.q, prob.kmax = warp + cta, warp, d, 1, 60 if cta else 30
    assert prob.kernel_launches(precision, chunked, est, nu) == kernels
