"""The shared-memory opt-in of a kernel (rspi_smem_optin) with callers of
different sizes on two threads: the attribute left behind serves both.  The
CUDA runtime's calls are replaced by host functions, of which the first
setter is held back until the other caller has returned."""
import os
import shutil
import subprocess

import pytest

from conftest import REPO

SOURCE = r'''
#include <cuda_runtime.h>
#include <atomic>
#include <chrono>
#include <cstdio>
#include <thread>

static std::atomic<int> attribute{49152}, setters{0}, other_done{0};
static std::thread::id first;

static cudaError_t fake_set(const void *, cudaFuncAttribute, int v) {
    setters++;
    if (std::this_thread::get_id() == first)
        for (int k = 0; k < 2000 && !other_done; ++k)
            std::this_thread::sleep_for(std::chrono::milliseconds(1));
    attribute = v;
    return cudaSuccess;
}
static cudaError_t fake_get(cudaFuncAttributes *a, const void *) {
    a->sharedSizeBytes = 1024;
    return cudaSuccess;
}
static cudaError_t fake_dev(int *v, cudaDeviceAttr, int) {
    *v = 232448;
    return cudaSuccess;
}
static cudaError_t fake_current(int *d) {
    *d = 0;
    return cudaSuccess;
}
#define cudaFuncSetAttribute fake_set
#define cudaFuncGetAttributes fake_get
#define cudaDeviceGetAttribute fake_dev
#define cudaGetDevice fake_current
#include "rspi_common.cuh"

int main() {
    static RspiSmemOptIn st;
    bool ok_small = false, ok_large = false;
    std::thread small([&] {
        first = std::this_thread::get_id();
        ok_small = rspi_smem_optin(&st, 30000, st);
    });
    while (setters == 0) std::this_thread::yield();
    std::thread large([&] {
        ok_large = rspi_smem_optin(&st, 100000, st);
        other_done = 1;
    });
    large.join();
    small.join();
    const bool again = rspi_smem_optin(&st, 100000, st);   // a later launch of the larger size
    const int left = attribute;
    const bool beyond = rspi_smem_optin(&st, 231425, st);
    printf("%d %d %d %d %d\n", ok_small, ok_large, again, left, beyond);
    return 0;
}
'''


@pytest.mark.skipif(shutil.which('nvcc') is None, reason='needs nvcc')
def test_optin_serves_concurrent_sizes(tmp_path):
    src, exe = str(tmp_path / 'optin.cu'), str(tmp_path / 'optin')
    with open(src, 'w') as f:
        f.write(SOURCE)
    subprocess.run(['nvcc', '-std=c++17', '-gencode', 'arch=compute_100a,code=sm_100a', '-I',
                    os.path.join(REPO, 'include'), '-I',
                    os.path.join(REPO, 'refspi-maxlp_b200', 'csrc'), src, '-o', exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, check=True, timeout=60).stdout
    small, large, again, attribute, beyond = map(int, out.split())
    assert small and large and again
    assert attribute >= 100000      # the larger launch's size is still allowed
    assert not beyond               # beside 1,024 static bytes
