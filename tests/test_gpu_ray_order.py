"""Memory of the ray order (batches of 2^14 to 2^22 rays on a refined octree):
an octree holds at most eight buffers however many threads and streams trace
through it, and a call that finds none free gives the same rays."""
import ctypes as C
import threading

import numpy as np
import pytest

from conftest import load_golden

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
PER_THREAD = 2      # cudaStreamPerThread: one handle, a stream of its own in every host thread


class Batch:
    """n rays on the device and a call on them without final or surface records."""

    def __init__(self, pkg, launch, length):
        from importlib import import_module
        self.capi = import_module(pkg.__name__ + ".capi")
        self.L = pkg.library()
        self.n = launch.shape[0]
        self.p, self.keep = self.capi.make_params(length, 2, 1, "redshift", 0.01, None, False, False, 0)
        self.launch = torch.from_numpy(np.ascontiguousarray(launch)).cuda()

    def out(self):
        return torch.zeros(self.n, dtype=torch.int64, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")

    def trace(self, tree, cos, steps, status, stream):
        self.capi.check(self.L.mpf_propagate_device(tree._h, cos._h, C.byref(self.p), self.n, C.c_void_p(self.launch.data_ptr()),
                                                    C.c_void_p(steps.data_ptr()), None, None, C.c_void_p(status.data_ptr()),
                                                    C.c_void_p(stream)))


@pytest.fixture(scope="module")
def cone(gpu_lib, pkg):
    g = load_golden("amr")
    tree = pkg.Octree.from_records(g["records"])
    cos = pkg.Cosmology(g["cosmo_t"], g["cosmo_a"], g["cosmo_dadt"], g["cosmo_d2adt2"])
    yield tree, cos, float(g["cosmo_length"])
    tree.close()
    cos.close()


def test_memory_does_not_grow_with_threads(cone, pkg, synth):
    """32 threads that live at the same time and trace one after the other, each
    on its own stream, a batch of 2^20 rays (4 MiB of order): the last 24 leave
    no more device memory in use than the first 8, but for one buffer (16 MiB)
    and what the threads' streams take."""
    tree, cos, length = cone
    batch = Batch(pkg, synth.photon_grid(1024, 2.4, 2.4), length)
    steps, status = batch.out()
    free, errors = [], []
    turn, done = threading.Lock(), threading.Event()

    def one():
        try:
            torch.cuda.set_device(0)
            with turn:
                batch.trace(tree, cos, steps, status, PER_THREAD)
                torch.cuda.synchronize()
                free.append(torch.cuda.mem_get_info()[0])
        except Exception as e:   # reported by the main thread
            errors.append(e)
        done.wait()              # a thread that ends gives its id to the next

    threads = [threading.Thread(target=one, daemon=True) for _ in range(32)]
    for t in threads:
        t.start()
    while len(free) + len(errors) < 32:
        threading.Event().wait(0.01)
    done.set()
    for t in threads:
        t.join()
    assert not errors, errors
    assert free[7] - free[-1] <= 32 << 20


def test_more_calls_in_flight_than_buffers(cone, pkg, synth):
    """Twelve streams with three calls each queued at once: every call gives the
    batch's rays."""
    tree, cos, length = cone
    batch = Batch(pkg, synth.photon_grid(182, 2.4, 2.4), length)      # 33 124 rays
    want, status = batch.out()
    batch.trace(tree, cos, want, status, 0)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(12)]
    calls = [(s, batch.out()) for _ in range(3) for s in streams]
    torch.cuda.synchronize()
    for s, (steps, st) in calls:
        batch.trace(tree, cos, steps, st, s.cuda_stream)
    torch.cuda.synchronize()
    assert int(want.min()) > 1
    for _, (steps, st) in calls:
        assert torch.equal(steps, want)
