"""A synchronous call returns when its results are there for everybody, whichever way the host waits for it: short calls, calls the host watches
a word for (norm layers of 2^16 elements and more), calls that outlast the watching, and what a capture on another stream forbids."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent
SHORT, WATCHED, LONG = (64, 64), (1024, 768), (65536, 4096)   # LayerNorm: a few us, a few us more, 350 us of memory traffic alone


class Norm:
    """LayerNorm through the function ids, its tensors seen by torch."""

    def __init__(self, cuda, rows, inner, seed):
        import torch
        self.cuda, self.n = cuda, rows * inner
        self.handle = cuda.CreateLayerNorm(0, self.n, 1, rows, inner, 1e-5)
        self.mem = [cuda.AllocMemory(self.n) for _ in range(2)]
        x, self.y = (torch.as_tensor(_View(cuda.GetPointer(m), self.n), device="cuda") for m in self.mem)
        x.normal_(generator=torch.Generator("cuda").manual_seed(seed))
        ref = torch.nn.functional.layer_norm(x.view(rows, inner), (inner,), eps=1e-5).view(-1)
        self.ref = ref
        self.side = torch.cuda.Stream()
        torch.cuda.synchronize()

    def check(self):
        """The call, then a read of its output on a stream that waits for no other."""
        import torch
        self.y.fill_(float("nan"))
        torch.cuda.synchronize()
        self.cuda.LayerNormForward(self.handle, *self.mem)
        with torch.cuda.stream(self.side):
            worst = float((self.y - self.ref).abs().max())   # nan where the output was not there yet
        assert worst < 1e-4

    def close(self):
        for m in self.mem:
            self.cuda.FreeMemory(m)
        self.cuda.FreeLayerNorm(self.handle)


class _View:
    def __init__(self, pointer, n):
        self.__cuda_array_interface__ = dict(shape=(n,), typestr="<f4", data=(pointer, False), version=3)


def calls_of_every_length():
    from mycaffe_b200 import CudaDnn
    for _ in range(2):                                # the second on the index that the first has given back
        cuda = CudaDnn(0)
        norms = [Norm(cuda, *shape, seed=i) for i, shape in enumerate((SHORT, WATCHED, LONG))]
        for _ in range(4):
            for i in (1, 2, 1, 0, 1):                 # a watched call directly behind one whose word came late
                norms[i].check()
        cuda.SetAsync(True)
        cuda.LayerNormForward(norms[2].handle, *norms[2].mem)   # work of asynchronous calls in front of a watched one
        cuda.SetAsync(False)
        norms[1].check()
        for n in norms:
            n.close()
        cuda.Dispose()


def test_results_are_there_for_streams_that_do_not_wait():
    calls_of_every_length()


def test_a_host_that_does_not_spin():
    """The same in a process whose device flags ask for blocking waits."""
    code = ("import ctypes, sys; import torch; torch.cuda.init();"
            "rt = ctypes.CDLL([l.split()[-1] for l in open('/proc/self/maps') if 'libcudart' in l][0]);"
            "assert rt.cudaSetDeviceFlags(4) == 0;"                                  # cudaDeviceScheduleBlockingSync
            "sys.path.insert(0, 'tests'); import test_synchronous_calls_gpu as t; t.calls_of_every_length(); print('done')")
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.split()[-1] == "done", r.stdout + r.stderr


@pytest.mark.parametrize("shape", [SHORT, WATCHED])
def test_a_capture_forbids_what_the_stream_synchronisation_forbids(shape):
    """While a stream of the thread captures in the global or the thread's mode, a call that waits is refused and the capture is
    invalid; in the relaxed mode both go through."""
    code = f"""
import ctypes as C, sys
sys.path.insert(0, 'tests')
import test_synchronous_calls_gpu as t
from mycaffe_b200 import CudaDnn
cuda = CudaDnn(0)
norm = t.Norm(cuda, *{shape}, seed=1)
norm.check()
rt = C.CDLL([l.split()[-1] for l in open('/proc/self/maps') if 'libcudart' in l][0])
for mode, name in enumerate(('global', 'thread_local', 'relaxed')):
    s, g = C.c_void_p(), C.c_void_p()
    assert rt.cudaStreamCreateWithFlags(C.byref(s), 1) == 0      # a stream that does not wait for the legacy one
    assert rt.cudaStreamBeginCapture(s, mode) == 0
    try:
        cuda.LayerNormForward(norm.handle, *norm.mem)
        answer = 'accepted'
    except Exception as e:
        answer = '900' if '[900]' in str(e) else str(e)
    print(name, answer, rt.cudaStreamEndCapture(s, C.byref(g)))
    try:
        cuda.LayerNormForward(norm.handle, *norm.mem)            # reports what the refused one left behind
    except Exception:
        pass
    rt.cudaGetLastError()
    norm.check()
"""
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.split("\n")[:3] == ["global 900 901", "thread_local 900 901", "relaxed accepted 0"], r.stdout
