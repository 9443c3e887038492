"""The tensor-core switch of the limb form (a test hook) holds for the thread that set it."""
import ctypes
import threading


def test_limb_tc_switch_is_the_threads_own(built_lib):
    f = built_lib.gbmmx_limb_tc
    f.argtypes, f.restype = [ctypes.c_int32], ctypes.c_int32
    old = f(1)
    seen = []

    def other():
        seen.append(f(0))
        seen.append(f(-1))

    t = threading.Thread(target=other)
    t.start()
    t.join()
    assert seen == [-1, 0]
    assert f(old) == 1
