"""What the packed Richards kernel issues to the FP64 pipe (clmgb/flops_model.py): the
operations of its source per level, apart from the divisions and powers on the integer
pipes, and their part of the roofline entry."""
import pytest

from clmgb import flops_model as fm


def test_operations_issued_to_the_fp64_pipe():
    # attempt: amx 1, bmx 3, cmx 1, rmx 1, bet 2, dwat 2, back substitution 2, error 2
    assert fm.fp64_operations(1, 0) == 1 + 3 + 1 + 1 + 2 + 2 + 2 + 2
    # refresh: water 2, hydraulic properties 5, fluxes and derivatives 11, net flux 2
    assert fm.fp64_operations(0, 1) == 2 + 5 + 11 + 2
    assert fm.integer_powers(5, 7) == 14
    assert fm.fp64_operations(1, 0) < fm.ATTEMPT["ops"] and fm.fp64_operations(0, 1) < fm.REFRESH["ops"]


def test_roofline_entry_names_them_apart():
    probe = (5.2e11, 7.0e10, 3.0e10, 4.0e10, 1.4e11)
    att, ref, launches, ms = 19.7e6 * 2, 15.2e6 * 2, 2, 3.84
    r = fm.fp64_roofline(att, ref, launches, ms, probe)
    assert r["fp64_operations_per_launch"] == pytest.approx(19.7e6 * 14 + 15.2e6 * 20)
    assert r["fp64_operations_frac"] == pytest.approx(r["fp64_operations_per_launch"] / (ms / 1e3) / probe[0])
    assert r["integer_pipe_powers_per_launch"] == pytest.approx(2 * 15.2e6)
    assert r["fp64_operations_frac"] < r["frac"]
