// State in and out of device planes: one kernel a call where the caller's planes are plain device memory, else a
// copy per plane.
//
// A copy per plane and the CFL scan behind them were eight stream operations to set a state and six to get it, at
// about 2.5 us each on the host and, between dependent copies, on the device: more than two small solves. The
// kernel that copies also takes the CFL maximum, so the state is read once (4096^2: 12 planes moved for 18).
// 24 instances of 48^2 .. 160^2 set, stepped four times and read: 1.88 -> 1.10 ms; 64 of 256^2 .. 1024^2, three
// steps: 13.6 -> 11.7 ms.
#pragma once

#include <cuda.h>

#include <cstdint>

#include "mhd_host_util.h"
#include "mhd_kernels.cuh"

namespace mhd {

// dst = src; st->smax_bits (zeroed before) = max CFL speed of src (as k_cfl_scan).
static __global__ void __launch_bounds__(256)
k_state_load(Domain D, CPlanes src, Planes dst, DeviceStatus* st) {
    __shared__ double red[32];
    const int nx = D.nx, ny = D.ny;
    double vmax = 0.0;
    for (int j = blockIdx.y; j < ny; j += gridDim.y)
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nx; i += gridDim.x * blockDim.x) {
        const size_t g = (size_t)j * nx + i;
        double u[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) u[k] = src.f[k][g];
        const double bxc = (u[4] + src.f[4][(size_t)j * nx + wrap(i + 1, nx)]) / 2.0;
        const double byc = (u[5] + src.f[5][(size_t)wrap(j + 1, ny) * nx + i]) / 2.0;
#pragma unroll
        for (int k = 0; k < 6; ++k) dst.f[k][g] = u[k];
        double rho = u[0];
        vmax = smax(vmax, cell_cfl_speed(rho, u[1], u[2], u[3], bxc, byc));
    }
    vmax = block_max<256>(vmax, red);
    if (threadIdx.x == 0) atomicMax(&st->smax_bits, (unsigned long long)__double_as_longlong(vmax));
}

// dst = src, plane by plane where dst is not null.
static __global__ void __launch_bounds__(256)
k_state_store(size_t n, CPlanes src, Planes dst) {
    for (size_t g = (size_t)blockIdx.x * blockDim.x + threadIdx.x; g < n; g += (size_t)gridDim.x * blockDim.x) {
        double u[6];
#pragma unroll
        for (int k = 0; k < 6; ++k)
            if (dst.f[k]) u[k] = src.f[k][g];
#pragma unroll
        for (int k = 0; k < 6; ++k)
            if (dst.f[k]) dst.f[k][g] = u[k];
    }
}

}  // namespace mhd

namespace mhd_host {

// A driver function, or null.
inline void* driver_entry(const char* name) {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPoint(name, &f, cudaEnableDefault, &found) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return found == cudaDriverEntryPointSuccess ? f : nullptr;
}

// Whether a kernel may use [p, p + bytes) as doubles: aligned memory of this device, inside one allocation, which is not
// another context's (pool memory is no context's). Anything else (host, managed, another context's or device's memory,
// ranges across allocations or too short) is left to the copy, which accepts or refuses it.
inline bool plain_device_range(const void* p, size_t bytes, int device) {
    using GetAttributes = CUresult (*)(unsigned int, CUpointer_attribute*, void**, CUdeviceptr);
    using GetCurrent = CUresult (*)(CUcontext*);
    static const GetAttributes get = (GetAttributes)driver_entry("cuPointerGetAttributes");
    static const GetCurrent current = (GetCurrent)driver_entry("cuCtxGetCurrent");
    const uintptr_t a = (uintptr_t)p;
    if (!get || !current || a % sizeof(double)) return false;
    unsigned int type = 0, managed = 1;
    int ordinal = -1;
    CUdeviceptr base = 0;
    size_t size = 0;
    CUcontext owner = nullptr, here = nullptr;
    CUpointer_attribute what[6] = {CU_POINTER_ATTRIBUTE_MEMORY_TYPE, CU_POINTER_ATTRIBUTE_IS_MANAGED,
                                   CU_POINTER_ATTRIBUTE_DEVICE_ORDINAL, CU_POINTER_ATTRIBUTE_RANGE_START_ADDR,
                                   CU_POINTER_ATTRIBUTE_RANGE_SIZE, CU_POINTER_ATTRIBUTE_CONTEXT};
    void* into[6] = {&type, &managed, &ordinal, &base, &size, &owner};
    if (get(6, what, into, (CUdeviceptr)a) != CUDA_SUCCESS || current(&here) != CUDA_SUCCESS) return false;
    return type == CU_MEMORYTYPE_DEVICE && !managed && ordinal == device && (!owner || owner == here) && base && a >= base &&
           a - base <= size && bytes <= size - (a - base);
}

// The six planes f (null: skipped) for a kernel that moves them to or from the planes s: plain memory, apart from
// s and, when written, from one another.
inline bool plain_state(const double* const* f, const double* const* s, size_t bytes, int device, bool written) {
    for (int k = 0; k < 6; ++k) {
        if (!f[k]) continue;
        for (int q = 0; q < 6; ++q)
            if (overlap(f[k], s[q], bytes) || (written && q < k && f[q] && overlap(f[k], f[q], bytes))) return false;
        if (!plain_device_range(f[k], bytes, device)) return false;
    }
    return true;
}

// s = f and its CFL speed into status.
static inline mhd_status load_state(const mhd::Domain& D, const double* const* f, double* const* s, mhd::DeviceStatus* status,
                             cudaStream_t stream) {
    MHD_TRY(cudaMemsetAsync(&status->smax_bits, 0, sizeof(unsigned long long), stream));
    mhd::CPlanes in;
    mhd::Planes out;
    for (int k = 0; k < 6; ++k) {
        in.f[k] = f[k];
        out.f[k] = s[k];
    }
    mhd::k_state_load<<<mhd::cell_grid(D.nx, D.ny), 256, 0, stream>>>(D, in, out, status);
    MHD_TRY(cudaGetLastError());
    return MHD_OK;
}

static inline mhd_status store_state(size_t n, const double* const* s, double* const* f, int num_sms, cudaStream_t stream) {
    mhd::CPlanes in;
    mhd::Planes out;
    for (int k = 0; k < 6; ++k) {
        in.f[k] = s[k];
        out.f[k] = f[k];
    }
    const size_t blocks = std::max<size_t>(1, std::min<size_t>((n + 255) / 256, (size_t)num_sms * 8));
    mhd::k_state_store<<<(unsigned)blocks, 256, 0, stream>>>(n, in, out);
    MHD_TRY(cudaGetLastError());
    return MHD_OK;
}

}  // namespace mhd_host
