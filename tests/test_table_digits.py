"""The digits of the reconstruction tables (csrc/crt.cu, build_tables_fit): base 256 where every
column's sum allows it, and one build to find that out."""
import ctypes

import pytest


@pytest.mark.parametrize("counts,bits", [
    ((1, 2, 300, 511, 512, 513, 738, 740, 780, 863, 884, 920, 921, 923, 926, 932, 939, 940), 8),
    ((739, 747, 748, 779, 786, 787, 788, 817, 823, 824, 825, 826, 848, 850, 853, 854, 859, 860, 861, 862, 883, 885, 888, 889,
      894, 895, 896, 897, 917, 919, 922, 927, 928, 929, 930, 931), 7),
    ((941, 1023), 7)])
def test_one_build(built_lib, counts, bits):
    f = built_lib.gbmmx_table_digits
    f.argtypes, f.restype = [ctypes.c_int32, ctypes.POINTER(ctypes.c_int32)], ctypes.c_int32
    for p in counts:
        n = ctypes.c_int32(0)
        assert (f(p, ctypes.byref(n)), n.value) == (bits, 1), p
