"""GPU test: the allocation-free multiply allocates nothing at a geometry that is set
after ffg_init either.  A fresh process sets row lengths and tile widths that no length
has by default or in the tuning file, one after another, and takes the device's free
memory around the first product at each."""
import os
import subprocess
import sys
import textwrap

import pytest

pytestmark = pytest.mark.gpu

_FRESH = textwrap.dedent("""
    import ctypes, sys
    import torch
    sys.path.insert(0, sys.argv[1])
    import fastfib_b200 as ff
    ff.set_device(0)
    torch.cuda.set_device(0)
    ff.init(1 << 20)
    f = ff.lib().ffg_mul_device_noalloc
    f.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_size_t, ctypes.c_uint64, ctypes.c_void_p,
                  ctypes.c_size_t, ctypes.c_uint64, ctypes.c_int, ctypes.c_void_p]
    a = torch.full((100000,), -1, dtype=torch.int64, device="cuda")
    out = torch.zeros(200001, dtype=torch.int64, device="cuda")
    runs = dropped = wrong = 0
    for lg in range(13, 18):
        for r3 in (0, 1):
            n = int((3 if r3 else 1) * 2**lg / 4 * 0.97)
            if ff.plan(64 * n, 64 * n, True)["L"] != (3 if r3 else 1) << lg:
                continue
            for c in range(8, 13):
                for wc in (8, 32):
                    try:
                        ff.set_geometry(lg, r3, c, wc)
                    except ff.FfgError:
                        continue
                    torch.cuda.synchronize()
                    free = torch.cuda.mem_get_info()[0]
                    assert f(out.data_ptr(), a.data_ptr(), n, 64 * n, a.data_ptr(), n, 64 * n, 1, None) == 0
                    torch.cuda.synchronize()
                    dropped += free - torch.cuda.mem_get_info()[0]
                    got = out[:2 * n + 1].cpu().numpy().tobytes()  # (2^(64 n) - 1)^2
                    wrong += int.from_bytes(got, "little") != (1 << 128 * n) - (1 << 64 * n + 1) + 1
                    runs += 1
    print(runs, dropped, wrong)
""")


def test_no_alloc_after_a_geometry_change():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _FRESH, root], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    runs, dropped, wrong = (int(v) for v in r.stdout.split()[-3:])
    assert runs >= 40 and wrong == 0
    assert dropped == 0, f"device free memory fell by {dropped} bytes during first calls"
