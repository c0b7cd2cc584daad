"""The step kernels' FP32 arithmetic that stands for IEEE division and the
double boundary mix (geopvi_gb300/csrc/fwi2d_exact.h), bit for bit on the CPU."""
import ctypes
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("step") / "libstep.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fno-fast-math", "-shared", "-fPIC",
                    "-o", out, os.path.join(HERE, "step_harness.cpp")], check=True)
    L = ctypes.CDLL(out)
    ll, f, i = ctypes.c_longlong, ctypes.c_float, ctypes.c_int
    L.harness_div_two.argtypes, L.harness_div_two.restype = [f, i, i], ll
    L.harness_div2_tiny.argtypes, L.harness_div2_tiny.restype = [f], ll
    L.harness_two_op_exact.argtypes = [f]
    L.harness_quotients_at_their_bounds.argtypes, L.harness_quotients_at_their_bounds.restype = [f], ll
    L.harness_div2_least.argtypes, L.harness_div2_least.restype = [f], f
    L.harness_mix.argtypes, L.harness_mix.restype = [i, ll, ctypes.c_uint, ctypes.POINTER(ll)], ll
    L.harness_mix_values.argtypes, L.harness_mix_values.restype = [i, ll, ctypes.c_uint, i], ll
    return L


@pytest.mark.parametrize("y", [10.0, 12.5, 8.0, 9.0, 20.0, 1.0])
def test_two_operation_quotient(harness, y):
    assert harness.harness_two_op_exact(y) == 1
    assert harness.harness_div_two(y, -100, -99) == 0  # the ends of its range and a middle binade
    assert harness.harness_div_two(y, -80, -80) == 0
    assert harness.harness_div_two(y, 0, 0) == 0
    assert harness.harness_div_two(y, 127, 127) == 0
    assert harness.harness_div2_least(y) <= 2.0 ** -100  # few bits: valid far below 2^-80
    assert harness.harness_div_two(y, -126, -101) == 0


def test_divisors_of_many_bits_keep_the_plain_range(harness):
    assert harness.harness_two_op_exact(8.4) == 1 and harness.harness_div2_least(8.4) == 2.0 ** -80
    assert harness.harness_div_two(8.4, -80, -79) == 0


def test_divisors_outside_the_proof_are_refused(harness):
    assert harness.harness_two_op_exact(11.7) == 0      # some significand rounds the other way
    assert harness.harness_two_op_exact(2.0 ** 21) == 0  # outside [2^-20, 2^20]


@pytest.mark.parametrize("y", [10.0, 12.5, 20.0, 8.4, 0.5, 2.0 ** -20, 2.0 ** 20])
def test_two_step_quotient_of_tails(harness, y):
    assert harness.harness_div2_tiny(y) == 0


@pytest.mark.parametrize("pml0", [1, 2, 5, 8, 10, 13, 20, 30])
def test_mix_matches_the_double_formula(harness, pml0):
    left, trials = ctypes.c_longlong(0), 64000
    assert harness.harness_mix(pml0, trials, 5 + pml0, ctypes.byref(left)) == 0
    # 5 of 16 trial kinds are tails, subnormals, ties and cancellations that may need the general path
    assert left.value <= 0.35 * trials * pml0


# Divisors of few and of many bits: where x times the reciprocal's low word turns subnormal, it no longer scales.
@pytest.mark.parametrize("y", [10.0, 12.3, 77.7, 9000.3, 25000.7, 0.37, 0.001, 4096.0, 2.0 ** 20])
def test_quotients_at_their_least_dividends(harness, y):
    assert harness.harness_quotients_at_their_bounds(y) == 0


@pytest.mark.parametrize("y", [12.3, 77.7, 25000.7])
def test_tails_of_divisors_of_many_bits(harness, y):
    assert harness.harness_div2_tiny(y) == 0


def test_divisors_whose_low_word_leaves_no_room_for_tails_are_refused(harness):
    assert harness.harness_two_op_exact(2500.3) == 1 and harness.harness_quotients_at_their_bounds(2500.3) == -1


@pytest.mark.parametrize("pml0", [1, 2, 8, 10, 13, 20, 40, 77, 300])  # from 33 on, some 1 - w have over 29 bits
def test_mix_by_value_matches_the_double_formula(harness, pml0):
    assert harness.harness_mix_values(pml0, max(4000, 640000 // pml0), 9 + pml0, 1 if pml0 <= 32 else 0) == 0
