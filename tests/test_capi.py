"""The C-ABI library loads and exports every function include/tictac_b200.h declares."""
import ctypes
import os
import re
import subprocess

import tictac_b200 as tt
from conftest import ROOT


def declared_functions():
    src = open(os.path.join(ROOT, "include", "tictac_b200.h")).read()
    src = re.sub(r"/\*.*?\*/", "", src, flags=re.S)
    return sorted(set(re.findall(r"\b(tt_[A-Za-z0-9_]+)\s*\(", src)))


def test_library_exports_every_declared_symbol():
    lib = tt.load()
    names = declared_functions()
    assert len(names) >= 30
    for name in names:
        assert hasattr(lib, name), f"{name} declared in include/tictac_b200.h but not exported"
    assert set(names) == set(tt.EXPORTED_SYMBOLS)


def test_error_paths_without_device():
    lib = tt.load()
    run = ctypes.c_void_p()
    bad = (ctypes.c_char_p * 1)(b"Np_WP")
    assert lib.tt_run_create(ctypes.byref(run), 1, bad) == tt.TT_ERR_BADARG
    assert b"=" in lib.tt_last_error_string()
    assert lib.tt_run_num_channels(None, None) == tt.TT_ERR_BADARG
    rp = tt.run_params()
    assert rp.Nphi == 48 and rp.Nx == 48 and rp.precision == tt.PRECISION_MIXED


def test_device_memory_is_written_in_stream_order():
    # the library's streams are non-blocking: a plain cudaMemcpy into device memory is
    # ordered with none of them, and from pageable memory may return before the data is there
    src = os.path.join(ROOT, "tic-tac_b200", "csrc")
    files = [os.path.join(d, f) for d, _, fs in os.walk(src) for f in fs if f.endswith((".cpp", ".cu", ".h", ".cuh"))]
    assert len(files) > 20
    for f in files:
        for call in re.findall(r"\bcudaMem(?:cpy|set)(?:2D)?\s*\([^;]*", open(f).read()):
            assert "cudaMemcpyDeviceToHost" in call, (f, call)


def compile_and_run(tmp_path, *sources):
    """main.cpp of tmp_path with sources of csrc, by the host compiler; the numbers it prints."""
    src, exe = os.path.join(ROOT, "tic-tac_b200", "csrc"), str(tmp_path / "main")
    cuda = os.environ.get("CUDA", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-I" + src, "-I" + os.path.join(ROOT, "include"), "-I" + cuda + "/include",
                    str(tmp_path / "main.cpp"), *(os.path.join(src, f) for f in sources), "-o", exe], check=True)
    return [int(x) for x in subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split()]


def test_a_failed_call_waits_for_its_stream(tmp_path):
    # the buffers' scope against a CUDA runtime of counters: what a failed call left queued
    # may use buffers that the next call frees on another stream
    (tmp_path / "main.cpp").write_text(r"""
#include <cstdio>
#include "cuda/tt_device.h"
static int waits = 0;
static unsigned long errors = 0;
namespace tt {
void set_error(const std::string&) { errors++; }
unsigned long error_count() { return errors; }
}
extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaMalloc(void**, size_t) { return cudaErrorMemoryAllocation; }
cudaError_t cudaFree(void*) { return cudaSuccess; }
cudaError_t cudaFreeAsync(void*, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { waits += s == (cudaStream_t)8; return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void**, size_t, cudaMemPool_t, cudaStream_t) { return cudaErrorMemoryAllocation; }
cudaError_t cudaMemPoolCreate(cudaMemPool_t*, const cudaMemPoolProps*) { return cudaErrorNotSupported; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemPoolGetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaErrorNotSupported; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) { return cudaSuccess; }
}
static void call(cudaStream_t st, bool fails) {
  tt::StreamScope scope(st);
  if (fails) tt::set_error("x");
}
int main() {
  call((cudaStream_t)8, false);
  const int good = waits;
  call((cudaStream_t)8, true);
  const int failed = waits;
  call(nullptr, true);
  { tt::StreamScope outer((cudaStream_t)8); call((cudaStream_t)16, true); }
  std::printf("%d %d %d", good, failed, waits);
}
""")
    assert compile_and_run(tmp_path, "host/tt_device_cache.cpp") == [0, 1, 2]


def test_subpanel_clusters(tmp_path):
    # rows of a sub-panel -> CTAs of its cluster, on devices whose largest cluster is 1, 8 or 16
    (tmp_path / "main.cpp").write_text(r"""
#include <cstdio>
#include "cuda/tt_lu_internal.h"
namespace tt { void set_error(const std::string&) {} }
int main() {
  for (int most : {1, 8, 16})
    for (size_t m : {224, 225, 256, 512, 513, 2048, 2049, 4096, 4097})
      std::printf("%d ", tt::subpanel_cluster_ctas(m, 224, 256, most));
}
""")
    assert compile_and_run(tmp_path) == [0] * 9 + [0, 2, 2, 2, 4, 8, 0, 0, 0] + [0, 2, 2, 2, 4, 8, 16, 16, 0]


def test_aligned_barriers_follow_a_converged_warp():
    # inline bar.sync, barrier.cluster.*.aligned and tcgen05.*.sync.aligned are undefined for
    # a warp whose lanes arrive apart, and the compiler does not converge it for them
    src = os.path.join(ROOT, "tic-tac_b200", "csrc", "cuda")
    found = 0
    for f in ("lu_factor.cu", "gemm_tc2.cu", "gemm_tc.cu"):
        text = open(os.path.join(src, f)).read()
        for m in re.finditer(r'asm volatile\(\s*"(bar\.sync|barrier\.cluster\.arrive|tcgen05\.(?:alloc|ld))', text):
            before = re.sub(r"//.*|if \(warp == 0\) \{", "", text[:m.start()]).rstrip()
            assert before.endswith("__syncwarp();"), (f, text.count("\n", 0, m.start()) + 1)
            found += 1
    assert found == 8


def test_changed_headers_rebuild_the_library():
    root = os.path.join(ROOT, "tic-tac_b200")
    headers = [os.path.join(d, f) for d, _, fs in os.walk(os.path.join(root, "csrc")) for f in fs
               if f.endswith((".h", ".cuh"))]
    assert len(headers) > 8
    for h in headers:
        out = subprocess.run(["make", "-n", "-C", root, "-W", h], capture_output=True, text=True, check=True).stdout
        assert ".cu " in out and " -shared " in out, h
