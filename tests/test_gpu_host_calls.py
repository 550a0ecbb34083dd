"""The host side of short calls: what a call may not ask of the allocator, and how often it
waits.  A preloaded library counts, for the calling thread, operator new and the runtime
calls of interest, and passes them on."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

import femm_gpu_b200 as fg
from conftest import ROOT
from femm_gpu_b200 import learned

pytestmark = pytest.mark.gpu

COUNTER = r"""
#include <cstdlib>
#include <dlfcn.h>
#include <new>
static thread_local bool on;
static thread_local long counts[3];
extern "C" void watch_start() { counts[0] = counts[1] = counts[2] = 0; on = true; }
extern "C" void watch_stop(long *out) { on = false; for (int i = 0; i < 3; ++i) out[i] = counts[i]; }
static void *real(const char *name) { return dlsym(dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD), name); }
void *operator new(std::size_t n)
{
  counts[0] += on;
  if (void *p = std::malloc(n ? n : 1))
    return p;
  throw std::bad_alloc();
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, std::size_t) noexcept { std::free(p); }
extern "C" int cudaMallocHost(void **p, std::size_t n)
{
  static auto f = reinterpret_cast<int (*)(void **, std::size_t)>(real("cudaMallocHost"));
  counts[1] += on;
  return f(p, n);
}
extern "C" int cudaStreamSynchronize(void *s)
{
  static auto f = reinterpret_cast<int (*)(void *)>(real("cudaStreamSynchronize"));
  counts[2] += on;
  return f(s);
}
"""

HEAD = """
import ctypes, numpy as np
import femm_gpu_b200 as fg
from femm_gpu_b200 import learned, meshes
watch = ctypes.CDLL(None)
counts = (ctypes.c_long * 3)()
def counted(call):
    watch.watch_start()
    try:
        call()
    finally:
        watch.watch_stop(counts)
    return list(counts)
"""


@pytest.fixture(scope="module")
def counter(tmp_path_factory):
    where = tmp_path_factory.mktemp("counter")
    source, library = where / "counter.cpp", where / "counter.so"
    source.write_text(COUNTER)
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", "-o", str(library), str(source), "-ldl"], check=True)

    def run(body):
        env = dict(os.environ, LD_PRELOAD=str(library), PYTHONPATH=os.path.join(ROOT, "femm-gpu_b200"))
        r = subprocess.run([sys.executable, "-c", HEAD + body], env=env, capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]

    return run


def test_the_counter_counts(gpu, counter):
    counter("""
new, pinned, waits = counted(lambda: fg.Plan(meshes.square_nonlinear(m=8, seed=1)).solve([[1.0, 2.0, 3.0]]))
assert new > 0 and pinned >= 0 and waits > 0, (new, pinned, waits)
""")


NOALLOC = """
import torch
model = meshes.square_nonlinear(m={m}, seed=12)
plan = fg.Plan(model)
ro, col, _, _, _ = plan.symbolic()
vals, diag, rhs = plan.assemble(np.zeros(plan.N), [3.0, -5.0, 8.0], 0)
bufs = [torch.tensor(x, device="cuda") for x in (ro, col, vals[0], diag[0], rhs[0])]
x = torch.zeros(plan.rows, dtype=torch.float64, device="cuda")
torch.cuda.synchronize()
def call():
    status, info = fg.capi.csr_pcg_noalloc(plan.rows, *[b.data_ptr() for b in bufs], x.data_ptr())
    assert status == 0 and info.status == 0
call()
new, pinned, waits = counted(call)
"""


@pytest.mark.parametrize("m", [20, 64])
def test_the_noalloc_solve_uses_no_heap(gpu, counter, m):
    counter(NOALLOC.format(m=m) + "assert new == 0 and pinned == 0, (new, pinned)")


@pytest.mark.parametrize("m", [20, 64])
def test_the_noalloc_solve_waits_three_times(gpu, counter, m):
    """For the set-up's verdict, for the solve's and for the copy of x."""
    counter(NOALLOC.format(m=m) + "assert waits == 3, waits")


def test_the_first_gradient_of_a_network_pins_no_memory(gpu, counter):
    counter("""
net = learned.Mlp(4, 64, 8, seed=1)
x, t = np.ones((16, 4), np.float32), np.ones((16, 8), np.float32)
new, pinned, waits = counted(lambda: net.loss_gradient(x, t))
assert pinned == 0, pinned
""")


def test_loss_and_gradient_are_the_same_wherever_the_loss_goes(gpu):
    """Behind the gradient (one copy), elsewhere, or only one of the two asked for."""
    net = learned.Mlp(4, 40, 5, seed=1)
    rng = np.random.default_rng(0)
    x, t = rng.normal(size=(24, 4)).astype(np.float32), rng.normal(size=(24, 5)).astype(np.float32)
    loss, g = net.loss_gradient(x, t)
    assert g.shape == (net.parameter_count,) and np.isfinite(loss) and loss > 0.0
    apart, alone = ctypes.c_float(0.0), ctypes.c_float(0.0)
    g2, g3 = np.zeros_like(g), np.zeros_like(g)
    ptr = lambda a: ctypes.c_void_p(a.ctypes.data)  # noqa: E731
    call = lambda loss, g: fg.lib().fg_mlp_loss_gradient(net._h, ctypes.c_int32(24), ptr(x), ptr(t), loss, g)  # noqa: E731
    assert call(ctypes.byref(apart), ptr(g2)) == call(ctypes.byref(alone), None) == call(None, ptr(g3)) == 0
    assert apart.value == alone.value == loss
    assert np.array_equal(g, g2) and np.array_equal(g, g3)
