// Conversions between the callers' host layouts (arrays of particles, blob arrays)
// and the device's, run on the device so that a call uploads and downloads the
// caller's memory as it is: no staging vectors, no loops over the blobs on the
// host.  All are a few passes over memory, far below the transfer's own time.
#include "dvm_internal.h"

namespace dvmk {
namespace {

__global__ void k_aos_to_soa(const double4* __restrict__ in, uint32_t m, double* __restrict__ out,
                             size_t n) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
        const double4 v = in[i];
        out[i] = v.x;
        out[n + i] = v.y;
        out[2 * n + i] = v.z;
        out[3 * n + i] = v.w;
    }
}

__global__ void k_pairs(const double* __restrict__ u, const double* __restrict__ w, uint32_t n,
                        double2* __restrict__ out) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        out[i] = make_double2(u[i], w[i]);
}

__global__ void k_soa_to_aos(const double* __restrict__ x, const double* __restrict__ z,
                             const double* __restrict__ c, const double* __restrict__ s,
                             const uint32_t* __restrict__ n, uint32_t first, uint32_t cap,
                             double4* __restrict__ out) {
    const uint32_t m = n[0] > first ? min(n[0] - first, cap) : 0u;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
        const size_t j = (size_t)first + i;
        out[i] = make_double4(x[j], z[j], c[j], s[j]);
    }
}

// Least index with a non-finite value in any of four arrays of n (bad starts at
// the largest value).
__global__ void k_check_finite(const double* __restrict__ v, uint32_t n, uint32_t* __restrict__ bad) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const bool ok = isfinite(v[i]) && isfinite(v[n + (size_t)i]) &&
                        isfinite(v[2 * (size_t)n + i]) && isfinite(v[3 * (size_t)n + i]);
        if (!ok) atomicMin(bad, i);
    }
}

// A checked blob set becomes the simulation's: positions, circulations, core sizes,
// zero velocities, IDs 0 .. n - 1 and the count; nothing when the check failed.
__global__ void k_take_blobs(const double* __restrict__ v, uint32_t n,
                             const uint32_t* __restrict__ bad, BlobArrays a, uint32_t* __restrict__ count) {
    if (*bad != UINT32_MAX) return;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        a.x[i] = v[i];
        a.z[i] = v[n + (size_t)i];
        a.circ[i] = v[2 * (size_t)n + i];
        a.sigma[i] = v[3 * (size_t)n + i];
        a.u[i] = a.w[i] = a.uvs[i] = a.wvs[i] = 0.0;
        a.id[i] = i;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) *count = n;
}

__global__ void k_fresh_blobs(uint32_t n, BlobArrays a, uint32_t* __restrict__ count) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        a.u[i] = a.w[i] = a.uvs[i] = a.wvs[i] = 0.0;
        a.id[i] = i;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) *count = n;
}

// Probe results: v = u, w, uvs, wvs of n points; u and w become the totals.
__global__ void k_probe_total(double* __restrict__ v, uint32_t n, double ux, double uz) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        v[i] = (v[i] + v[2 * (size_t)n + i]) + ux;
        v[n + (size_t)i] = (v[n + (size_t)i] + v[3 * (size_t)n + i]) + uz;
    }
}

__global__ void k_setup_slot(InstDesc* d, InstDesc dv, InstState* st, InstState sv, ListEntry* e,
                             ListEntry ev) {
    *d = dv;
    *st = sv;
    *e = ev;
}

unsigned blocks_for(uint64_t n) {
    return (unsigned)((n + 255) / 256 < 1184 ? (n + 255) / 256 : 1184);
}

}  // namespace

void aos_to_soa(const void* in, uint32_t m, double* out, uint64_t n, cudaStream_t s) {
    if (m) k_aos_to_soa<<<blocks_for(m), 256, 0, s>>>(static_cast<const double4*>(in), m, out, n);
}

void velocity_pairs(const double* u, const double* w, uint32_t n, void* out, cudaStream_t s) {
    if (n) k_pairs<<<blocks_for(n), 256, 0, s>>>(u, w, n, static_cast<double2*>(out));
}

void soa_to_aos(const double* x, const double* z, const double* c, const double* sg,
                const uint32_t* n, uint32_t first, uint32_t cap, void* out, cudaStream_t s) {
    if (cap)
        k_soa_to_aos<<<blocks_for(cap), 256, 0, s>>>(x, z, c, sg, n, first, cap, static_cast<double4*>(out));
}

void take_blobs(const double* v, uint32_t n, uint32_t* bad, const BlobArrays& a, uint32_t* count,
                cudaStream_t s) {
    cudaMemsetAsync(bad, 0xff, sizeof(uint32_t), s);
    if (n) k_check_finite<<<blocks_for(n), 256, 0, s>>>(v, n, bad);
    k_take_blobs<<<n ? blocks_for(n) : 1, 256, 0, s>>>(v, n, bad, a, count);
}

void fresh_blobs(uint32_t n, const BlobArrays& a, uint32_t* count, cudaStream_t s) {
    k_fresh_blobs<<<n ? blocks_for(n) : 1, 256, 0, s>>>(n, a, count);
}

void probe_total(double* v, uint32_t n, double ux, double uz, cudaStream_t s) {
    if (n) k_probe_total<<<blocks_for(n), 256, 0, s>>>(v, n, ux, uz);
}

void setup_slot(InstDesc* d, const InstDesc& dv, InstState* st, const InstState& sv, ListEntry* e,
                const ListEntry& ev, cudaStream_t s) {
    k_setup_slot<<<1, 1, 0, s>>>(d, dv, st, sv, e, ev);
}

}  // namespace dvmk
