"""Kernel attributes and limits hold per device: the host code that asks for
them, compiled against a stand-in of the CUDA runtime with several devices."""

import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "solvcon_gb300", "csrc")

RUNTIME = r"""
#include <cuda_runtime_api.h>

#include <map>

static int g_device = 0;
static int g_largest[6] = {16, 16, 8, 4, 1, 0}; // cluster that each device schedules
static int g_calls = 0;
static std::map<int, int> g_shared, g_wide; // by device
static bool g_refuse = false;
static cudaError_t g_last = cudaSuccess;

extern "C"
{
cudaError_t cudaGetDevice(int * dev)
{
    *dev = g_device;
    return cudaSuccess;
}
cudaError_t cudaGetLastError()
{
    cudaError_t const rc = g_last;
    g_last = cudaSuccess;
    return rc;
}
cudaError_t cudaPeekAtLastError() { return g_last; }
char const * cudaGetErrorString(cudaError_t) { return "refused"; }
cudaError_t cudaFuncSetAttribute(void const *, cudaFuncAttribute attr, int value)
{
    if (g_refuse)
    {
        return g_last = cudaErrorInvalidValue;
    }
    ++g_calls;
    (attr == cudaFuncAttributeMaxDynamicSharedMemorySize ? g_shared : g_wide)[g_device] = value;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int * n, void const *, cudaLaunchConfig_t const * cfg)
{
    int const size = static_cast<int>(cfg->attrs[0].val.clusterDim.x);
    if ((size > 8 && !g_wide[g_device]) || size > 2 * g_largest[g_device])
    {
        return g_last = cudaErrorInvalidClusterSize;
    }
    *n = size <= g_largest[g_device] ? 1 : 0;
    return cudaSuccess;
}
void ** __cudaRegisterFatBinary(void *) { return nullptr; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}

void use(int device) { g_device = device; }
void refuse(int on) { g_refuse = on != 0; }
int shared_of(int device) { return g_shared[device]; }
int wide_of(int device) { return g_wide[device]; }
int calls() { return g_calls; }
}
"""

HOST = r"""
#include "cluster.cuh"
#include "euler_core.hpp"

namespace scg
{
std::atomic<int64_t> g_launches{0}, g_device_allocs{0};
}

static void kernel_a(int) {}
static void kernel_b(int) {}

extern "C" int fits(int64_t threads)
{
    int blocks = 0, warps = 0;
    return scg::cluster::cluster_shape<kernel_a, 4>(threads, blocks, warps) ? blocks * warps : 0;
}
extern "C" int limit() { return scg::cluster::cluster_limit<kernel_a, 128>(); }
extern "C" int allow()
{
    try
    {
        scg::allow_shared<kernel_b, 65536>();
        return 0;
    }
    catch (scg::CudaError const &)
    {
        return 1;
    }
}
"""


@pytest.fixture()
def host(tmp_path):
    from solvcon_gb300.build import nvcc
    if not os.path.exists(nvcc()):
        pytest.skip("no nvcc")
    files, out = [], str(tmp_path / "host.so")
    for name, text in (("runtime.cpp", RUNTIME), ("host.cu", HOST)):
        files.append(str(tmp_path / name))
        with open(files[-1], "w") as f:
            f.write(text)
    subprocess.run([nvcc(), "-std=c++17", "-O1", "-shared", "--cudart", "none",
                    "-gencode=arch=compute_103a,code=sm_103a", "-Xcompiler",
                    "-fPIC", "-Xlinker", "-Bsymbolic", "-I" + CSRC, "-o", out]
                   + files, check=True)
    return ctypes.CDLL(out)


def test_attributes_are_set_on_every_device(host):
    """The permission for a cluster of 16 blocks and for more than 48 KB of
    dynamic shared memory is asked for on each device, once."""
    for dev in (0, 1):
        host.use(dev)
        assert host.limit() == 16 and host.wide_of(dev) == 1
        assert host.allow() == 0 and host.shared_of(dev) == 65536
    host.use(2)
    assert host.limit() == 8
    before = host.calls()
    for dev in (0, 1, 2, 1, 0):
        host.use(dev)
        assert host.limit() == (8 if dev == 2 else 16)
        assert dev == 2 or host.allow() == 0
    assert host.calls() == before


def test_a_refusal_is_reported_and_asked_again(host):
    host.refuse(1)
    assert host.allow() == 1 and host.allow() == 1
    host.refuse(0)
    assert host.allow() == 0 and host.shared_of(0) == 65536


@pytest.mark.parametrize("dev,size", [(0, 16), (2, 8), (3, 4), (4, 1), (5, 0)])
def test_no_cluster_is_larger_than_the_device_schedules(host, dev, size):
    """A march takes one cluster only where its threads fit the largest one,
    four warps to a block, and none where the device schedules none."""
    host.use(dev)
    host.fits.argtypes = [ctypes.c_int64]
    assert host.limit() == size
    assert host.fits(size * 128) == 4 * size
    assert host.fits(size * 128 + 1) == 0
    assert host.cudaPeekAtLastError() == 0  # what the next launch looks at
