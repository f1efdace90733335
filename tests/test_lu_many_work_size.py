"""CPU: the workspace that mpdok_lu_ir_many_work_size reports covers every pass of the solve."""
import pytest


def _passes(nrhs):
    """Column counts of the passes of mpdok_lu_ir_solve_many: up to 16 groups of eight, then the remainder."""
    out = []
    while nrhs >= 8:
        out.append(min(128, nrhs // 8 * 8))
        nrhs -= out[-1]
    return out + ([nrhs] if nrhs else [])


@pytest.mark.parametrize("nrhs", [1, 7, 8, 11, 72, 127, 128, 129, 135, 136, 141, 200, 231, 248, 256, 263, 1000])
def test_size_covers_each_pass(native_lib, nrhs):
    """A pass of fewer columns may split K further and so need more partial sums:
    n = 4500 takes one piece for 128 columns and four for the 72 that follow."""
    lib = native_lib
    for n in [1, 300, 2047, 2048, *range(2100, 33000, 271), 4500, 7000, 32768]:
        have = lib.mpdok_lu_ir_many_work_size(n, nrhs)
        for k in set(_passes(nrhs)):
            assert have >= lib.mpdok_lu_ir_many_work_size(n, k), (n, k)
            if k <= 8:
                assert have >= lib.mpdok_lu_ir_multi_work_size(n, k), (n, k)
