"""The device norms' workspace over the life of Envs, threads and contexts.

The built-in problem's norms are exact integers below 2^53: every call gives
the same two numbers whatever else runs."""
import os
import subprocess
import sys
import textwrap
import threading

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import minisweep_b200 as msb  # noqa: E402

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
FLAGS = "--ncell_x 9 --ncell_y 8 --ncell_z 7 --ne 5 --na 16"


def test_norms_after_a_device_reset():
    """A host program may end its CUDA context between two Envs: in a child
    process without torch, nothing of the library may outlive the reset."""
    child = textwrap.dedent(f"""
        import ctypes
        import minisweep_b200 as msb
        msb.lib()
        rt = ctypes.CDLL("libcudart.so.12")
        rt.cudaMalloc.argtypes = [ctypes.POINTER(ctypes.c_void_p), ctypes.c_size_t]
        got = []
        for k in range(3):
            pb = msb.Problem({FLAGS!r}, nm=8)
            v = [ctypes.c_void_p(), ctypes.c_void_p()]
            for p in v:
                assert rt.cudaMalloc(ctypes.byref(p), 8 * pb.nstate) == 0
            pb.init_state_device(v[0].value)
            pb.sweep_device(v[1].value, v[0].value)
            got += [pb.norms_device(v[0].value, v[1].value) for _ in range(2)]
            pb.close()
            assert rt.cudaDeviceReset() == 0
        assert len(set(got)) == 1 and got[0][0] > 0 and got[0][1] == 0.0, got
        print("ok")
    """)
    r = subprocess.run([sys.executable, "-c", child], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stderr[-2000:]


def test_norms_while_other_envs_come_and_go():
    """Two threads take norms on Envs of their own while a third opens and
    finalises Envs, each of which gives the kept workspace back."""
    stop = threading.Event()
    bad, n = [], [0, 0]

    def norms(k):
        try:
            with msb.Problem(FLAGS, nm=8) as pb:
                vi = torch.empty(pb.nstate, dtype=torch.float64, device="cuda")
                vo = torch.empty_like(vi)
                torch.cuda.synchronize()
                pb.init_state_device(vi.data_ptr())
                pb.sweep_device(vo.data_ptr(), vi.data_ptr())
                first = pb.norms_device(vi.data_ptr(), vo.data_ptr())
                assert first[0] > 0 and first[1] == 0.0
                while not stop.is_set() or n[k] < 20:
                    assert pb.norms_device(vi.data_ptr(), vo.data_ptr()) == first
                    n[k] += 1
        except Exception as e:  # reported by the main thread
            bad.append(e)

    ts = [threading.Thread(target=norms, args=(k,)) for k in range(2)]
    for t in ts:
        t.start()
    for _ in range(20):
        with msb.Problem(FLAGS, nm=8) as pb:
            v = torch.zeros(pb.nstate, dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
            assert pb.norms_device(v.data_ptr(), v.data_ptr()) == (0.0, 0.0)
    stop.set()
    for t in ts:
        t.join(120)
    assert not bad and min(n) >= 20, (bad, n)
