"""The form that a launch of the FP32 attention takes (csrc/mha_f32_plan.h, plain C++)."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tensorrt_b200", "csrc")
SMS = 148


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("f32plan")
    (d / "plan.cpp").write_text('#include "mha_f32_plan.h"\n'
                                'extern "C" void plan(int32_t B, int32_t N, int32_t S, int32_t d, int32_t full, int64_t sms, int32_t* out)'
                                "{ auto p = b200::planAtt(B, N, S, d, full, sms); out[0] = p.rows; out[1] = p.perSm; out[2] = p.async; out[3] = p.skip; }\n")
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", f"-I{CSRC}", str(d / "plan.cpp"), "-o", str(d / "plan.so")], check=True)
    so = ctypes.CDLL(str(d / "plan.so"))

    def call(b, n, s, d=64, full=0):
        out = (ctypes.c_int32 * 4)()
        so.plan(b, n, s, d, full, ctypes.c_int64(SMS), out)
        assert out[3] or (full and s % 64 == 0 and out[0] == 64 and not out[2])   # keys are only kept where there are none to leave out
        return out[0], out[1], bool(out[2])

    return call


def _rounds(pairs, s, rows):
    return -(-pairs * -(-s // rows) // SMS)   # CTAs per SM, the fullest


@pytest.mark.parametrize("head_size", [32, 64])
def test_every_launch_fits_the_residency_it_asks_for(plan, head_size):
    """A limit of CTAs per SM never makes a second round; 32 rows only where they take half the time of 64 less a round, or fill their rows better."""
    for pairs in list(range(1, 320)) + [444, 445, 592, 600, 888, 1000, 1776, 5000]:
        for s in (1, 16, 32, 33, 64, 65, 96, 97, 128, 129, 192, 193, 200, 256, 257, 400, 512, 1000):
            rows, per_sm, asynchronous = plan(pairs, 1, s, head_size)
            assert plan(pairs, 1, s, head_size, 1) == (rows, per_sm, asynchronous)
            n64, n32 = _rounds(pairs, s, 64), _rounds(pairs, s, 32)
            assert rows in (32, 64) and per_sm in (0, 1, 2, 3)
            if per_sm:
                assert per_sm == (n32 if rows == 32 else n64)
            if rows == 32:
                assert asynchronous and n32 <= 2 * n64 - 2
            else:
                assert n32 > 2 * n64 - 2 or n64 > 6
                assert asynchronous == (head_size == 64 and s <= 128)


def test_examples(plan):
    assert plan(8, 12, 128) == (64, 2, True)     # 192 CTAs of 64 rows: 384 of 32 would be three per SM
    assert plan(7, 12, 200) == (32, 0, True)     # 336 of 64 rows are three per SM, 588 of 32 four
    assert plan(5, 16, 65) == (32, 2, True)
    assert plan(4, 12, 256) == (64, 2, False)
    assert plan(16, 12, 256) == (64, 0, False)
    assert plan(100, 12, 16) == (32, 0, True)    # 64 rows would be three quarters empty
    assert plan(1, 12, 16) == (64, 1, True)
    assert plan(8, 12, 128, 32) == (64, 2, False)
