"""GPU tests of a solve's order on its stream when the caller's own kernels are
programmatic dependent launches: a solve starts after every kernel queued
before it, and what is queued after a call starts after that call's last pass.

The caller's kernels are compiled here: `late` lets its dependents start at
once, waits on the clock for some milliseconds and writes the field; `next`,
launched as its dependent, lets its own dependents start at once and waits for
`late`; `copy` is launched as a dependent of a call that lets none start early,
and so does not wait on the device."""
import ctypes
import subprocess

import pytest

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include <cuda_runtime.h>
__device__ long long now() { long long t; asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t)); return t; }
__global__ void k_late(double *f, const double *src, long n, long long ns) {
  asm volatile("griddepcontrol.launch_dependents;");
  const long long t0 = now();
  for (int i = 0; i < 100000 && now() - t0 < ns; i++) __nanosleep(1000);
  for (long q = blockIdx.x * (long)blockDim.x + threadIdx.x; q < n; q += (long)gridDim.x * blockDim.x) f[q] = src[q];
}
__global__ void k_next() { asm volatile("griddepcontrol.launch_dependents;\n\tgriddepcontrol.wait;" ::: "memory"); }
__global__ void k_copy(double *out, const double *src, long n) {
  for (long q = blockIdx.x * (long)blockDim.x + threadIdx.x; q < n; q += (long)gridDim.x * blockDim.x) out[q] = src[q];
}
template <typename... P, typename... A> static int go(int dependent, void (*k)(P...), unsigned grid, void *st, A... a) {
  cudaLaunchConfig_t c{};
  c.gridDim = dim3(grid);
  c.blockDim = dim3(256);
  c.stream = static_cast<cudaStream_t>(st);
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &attr;
  c.numAttrs = dependent;
  return (int)cudaLaunchKernelEx(&c, k, static_cast<P>(a)...);
}
extern "C" int late(double *f, const double *src, long n, long long ns, int with_next, void *st) {
  const int rc = go(0, k_late, 8, st, f, src, n, ns);
  return rc || !with_next ? rc : go(1, k_next, 1, st);
}
extern "C" int dependent_copy(double *out, const double *src, long n, void *st) {
  return go(1, k_copy, 32, st, out, src, n);
}
"""


@pytest.fixture(scope="module")
def caller(tmp_path_factory):
    from fishfry_b200 import build
    d = tmp_path_factory.mktemp("caller")
    (d / "caller.cu").write_text(SOURCE)
    subprocess.run([build._nvcc()] + build.ARCH + ["-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-o", str(d / "caller.so"),
                    str(d / "caller.cu")], check=True)
    L = ctypes.CDLL(str(d / "caller.so"))
    L.late.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_long, ctypes.c_longlong, ctypes.c_int, ctypes.c_void_p]
    L.dependent_copy.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_long, ctypes.c_void_p]
    return L


# z passes of each kind: compile-time, generic, Rader's, Bluestein's
GRIDS = [(64, 64, 64), (30, 45, 50), (32, 32, 41), (32, 32, 46)]


@pytest.mark.parametrize("n", GRIDS)
def test_solve_starts_after_all_earlier_kernels(torch_cuda, ff, caller, n):
    torch = torch_cuda
    plan = ff.Plan(n)
    size, N = plan.nbytes // 8, n[0] * n[1] * n[2]
    f = torch.randn(N, dtype=torch.float64, device="cuda")
    d, p = (torch.zeros(size, dtype=torch.float64, device="cuda") for _ in range(2))
    d[:N] = f
    plan.solve(d, p)
    want = p[:N].clone()
    assert bool(want.any())
    st = torch.cuda.current_stream().cuda_stream
    for with_next in (0, 1, 0, 1):
        d.zero_()
        p.zero_()
        torch.cuda.synchronize()
        assert caller.late(d.data_ptr(), f.data_ptr(), N, 3_000_000, with_next, st) == 0
        plan.solve(d, p)
        torch.cuda.synchronize()
        assert torch.equal(p[:N], want)


@pytest.mark.parametrize("passes", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("n", [(128, 128, 128), (100, 90, 80), (113, 127, 89)])
def test_what_follows_a_call_starts_after_its_last_pass(torch_cuda, ff, caller, n, passes):
    torch = torch_cuda
    plan = ff.Plan(n)
    size, N = plan.nbytes // 8, n[0] * n[1] * n[2]
    f = torch.randn(N, dtype=torch.float64, device="cuda")
    d, p = (torch.zeros(size, dtype=torch.float64, device="cuda") for _ in range(2))
    out = torch.zeros_like(d)
    res = d if passes == 4 else p
    st = torch.cuda.current_stream().cuda_stream
    for _ in range(3):
        d[:N] = f
        torch.cuda.synchronize()
        plan.solve_passes(d, p, passes)
        assert caller.dependent_copy(out.data_ptr(), res.data_ptr(), size, st) == 0
        torch.cuda.synchronize()
        assert torch.equal(out[:N], res[:N])
