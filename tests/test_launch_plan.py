"""CPU: icbc_gpu_launch_plan refuses arguments that no image has."""
import ctypes

import icbc_gb300 as ig


def test_invalid_arguments():
    lib, info = ig.load(), ig.LaunchInfo()
    for level, w, h, mode in ((-1, 4, 4, 0), (10, 4, 4, 0), (3, 0, 4, 0), (3, 4, -1, 0), (3, 4, 4, 3)):
        assert lib.icbc_gpu_launch_plan(level, w, h, mode, ctypes.byref(info)) == 1
    assert lib.icbc_gpu_launch_plan(3, 4, 4, 0, None) == 1
