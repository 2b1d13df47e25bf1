"""The rule that deals an SM's shared memory out to the matrix-instruction GEMV (csrc/gemv_kquant.cu plan_teams): every shape that the kernel accepts has at
least one stage for each team.  Host code only."""
import ctypes as C

import pytest

from ntransformer_b200._lib import lib
from ntransformer_b200.dtypes import DType

FORMATS = [(DType.Q4_K_M,), (DType.Q5_K,), (DType.Q6_K,), (DType.Q8_0,), (DType.Q4_0,)]
MIXES = [(DType.Q4_K_M, DType.Q4_K_M, DType.Q6_K), (DType.Q4_K_M, DType.Q5_K), (DType.Q4_0, DType.Q6_K), (DType.Q5_K, DType.Q6_K, DType.Q8_0)]
# bytes of a 16-row stage for teams of 4, 8, 16 warps (two super-blocks to a warp in teams of 4 where the blocks are small), of an odd number of units
BLOCK = {DType.Q4_K_M: 144, DType.Q5_K: 176, DType.Q6_K: 210, DType.Q8_0: 272, DType.Q4_0: 144}


def stage(dt, kw):
    blocks = 2 * kw if kw == 4 and dt not in (DType.Q6_K, DType.Q8_0) else kw
    return 16 * ((((blocks * BLOCK[dt] + 15) // 16 + (dt == DType.Q6_K)) | 1) * 16)


def plan(dts, rows, cols, epilogue=0, whole=0):
    n, out = len(dts), (C.c_int * 4)()
    rc = lib().nt_b200_gemv_fused_plan(n, (C.c_int * n)(*[rows] * n), (C.c_int * n)(*map(int, dts)), cols, epilogue, whole, out)
    return rc, tuple(out)


@pytest.mark.parametrize("dts", FORMATS + MIXES, ids=lambda d: "+".join(x.name for x in d))
def test_every_accepted_shape_has_a_stage(dts):
    one = dts if set(dts) != {DType.Q5_K, DType.Q6_K, DType.Q8_0} and set(dts) != {DType.Q4_0, DType.Q6_K} else dts[:1]      # mixes without a kernel: one launch each
    for cols in range(256, 49152 + 1, 256):
        for rows in (1, 16, 148 * 16, 148 * 16 + 1, 256 * 16, 256 * 16 + 1, 128256):
            for epilogue in (0, 2) if len(dts) == 2 else (0,):
                rc, (kw, teams, stages, digits) = plan(dts, rows, cols, epilogue)
                assert rc == 0 and (kw, teams) in ((4, 4), (8, 2), (16, 1), (8, 1)) and 1 <= stages <= 8, (dts, cols, rows)
                assert digits == 3
                # digit planes, scales and sums of the vector, and the rings, in the 227 KB of a CTA
                assert 3 * (cols + 64) + cols // 4 + teams * stages * max(stage(d, kw) for d in one) <= 227 * 1024 - 4000, (dts, cols, rows)


def test_whole_activations():
    """launch_gemv of Q4_0 asks for four digits: there where a stage is left beside them, which the launcher checks"""
    for cols in range(256, 49152 + 1, 256):
        for rows in (1, 148 * 16 + 1, 256 * 16 + 1, 128256):
            rc, (kw, teams, stages, digits) = plan((DType.Q4_0,), rows, cols, whole=1)
            assert rc == 0 and stages >= 1 and (digits == 4 or cols > 28672)
            assert digits * (cols + 64) + (cols // 4 if digits == 3 else cols * 3 // 8) + teams * stages * stage(DType.Q4_0, kw) <= 227 * 1024 - 4000
            assert plan((DType.Q6_K,), rows, cols, whole=1)[1][3] == 3


def test_longer_rows_are_refused():
    assert plan((DType.Q4_K_M,), 4096, 49152 + 256)[0] == -2
    assert plan((DType.Q4_K_M,), 4096, 128)[0] == -2
    assert plan((DType.F16,), 4096, 4096)[0] == -2


# us call after call in teams of 4 (one stage), in teams of 8
@pytest.mark.parametrize("dt,rows,cols,whole,want", [
    (DType.Q8_0, 14529, 27904, 0, (4, 4, 1)),       # 103.8, 112.9 with one stage
    (DType.Q8_0, 6000, 36096, 0, (4, 4, 1)),        # 68.4, 74.1
    (DType.Q6_K, 14529, 48128, 0, (4, 4, 1)),       # 207.6, 224.5
    (DType.Q8_0, 4113, 27904, 0, (8, 2, 1)),        # 51.3, 35.6: one round
    (DType.Q8_0, 14529, 26624, 0, (8, 2, 2)),       # 97.9, 74.0
    (DType.Q6_K, 14529, 35840, 0, (8, 2, 2)),       # 157.1, 106.0
    (DType.Q4_K_M, 8192, 28672, 0, (8, 2, 3)),      # 41.1, 35.5
    (DType.Q5_K, 14529, 41472, 0, (8, 2, 2)),       # 112.9, 107.0
    (DType.Q4_0, 8192, 36096, 1, (8, 2, 1)),        # 1217 in the generic form, for want of the fourth digit, 72
    (DType.Q6_K, 8192, 28672, 0, (4, 4, 2)),
])
def test_long_rows_take_the_faster_teams(dt, rows, cols, whole, want):
    rc, out = plan((dt,), rows, cols, whole=whole)
    assert rc == 0 and out[:3] == want
