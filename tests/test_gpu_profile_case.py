"""The profiled workload of one bench step refines to its tolerance: the residual reads
A's values from the caller's device array, which must live as long as the factor (40^3:
large enough for the allocator to hand a freed array's memory to the right-hand
sides)."""
import pytest


@pytest.mark.gpu
def test_factor_refine_workload_converges(tb, capsys):
    from taucs_b200 import profile_case
    profile_case.main(["profile_case", "factor-refine", "40"])
    words = capsys.readouterr().out.split()
    assert 0 <= int(words[2]) <= 10 and float(words[-1]) <= 1e-12, words
