"""Kernels of more than 48 KiB of shared memory, launched from one process on two devices.  No GPU: the sources are compiled against
a device that only keeps count, where (as on a real one) a kernel's limit is raised for the current device alone."""
import ctypes
import subprocess

import pytest

from lgml_b200 import csrc

FAKE = r"""
#include <cuda_runtime.h>
#include <set>
#include <utility>
static int fake_device, fake_large, fake_refused;
static std::set<std::pair<int, const void *>> fake_raised;
template <typename K> cudaError_t fake_set(K kernel, cudaFuncAttribute, int) { return fake_raised.insert({fake_device, (const void *)kernel}), cudaSuccess; }
template <typename K, typename... A> cudaError_t fake_launch(const cudaLaunchConfig_t *cfg, K kernel, A &&...) {
    if (cfg->dynamicSmemBytes <= 48 * 1024) return cudaSuccess;
    ++fake_large, fake_refused += !fake_raised.count({fake_device, (const void *)kernel});
    return cudaSuccess;
}
extern "C" __attribute__((visibility("default"))) int fake_count(int device, int refused) { return fake_device = device, refused ? fake_refused : fake_large; }
#define cudaFuncSetAttribute fake_set
#define cudaLaunchKernelEx fake_launch
#define cudaGetLastError() cudaSuccess
"""


def gemm(lib, p):
    for m, n, k in ((16, 5000, 512), (1000, 2000, 64)):
        yield lib.lgml_gemm_f32(p, p, p, p, 0, m, n, k, k, k, n, p)


def attention(lib, p):
    f = ctypes.c_float
    for n_tiles, n_chunks in ((3, 0), (0, 4)):
        yield lib.lgml_attention_f32(p, 2048, p, p, p, n_tiles, p, 9, p, 9, p, p, 90, 64, p, 2048, 16, 4, 128, f(0.1), 0, f(0.0), n_chunks, 9, p, p, p, p)


@pytest.mark.parametrize("name,calls", [("gemm_f32", gemm), ("attention_f32", attention)])
def test_large_kernels_run_on_every_device_of_a_process(tmp_path, name, calls):
    (tmp_path / "fake.h").write_text(FAKE)
    out = tmp_path / "lib.so"
    cmd = [csrc.find_nvcc(), "-gencode", "arch=compute_100a,code=compute_100a", "-Xcicc", "-O0", "-std=c++17", "--shared", "-Xcompiler", "-fPIC",
           "-include", str(tmp_path / "fake.h"), "-I", str(csrc.HERE), str(csrc.HERE / csrc.LIBRARIES[name][0]), "-o", str(out)]
    done = subprocess.run(cmd, capture_output=True, text=True)
    assert done.returncode == 0, done.stderr
    lib = ctypes.CDLL(str(out))
    for device in (0, 1):
        before = lib.fake_count(device, 0)
        assert all(rc == 0 for rc in calls(lib, ctypes.c_void_p(0x1000)))
        assert lib.fake_count(device, 0) > before          # there were such launches
    assert lib.fake_count(1, 1) == 0
