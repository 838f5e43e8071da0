// dem_records.cuh -- contact records and forces on their way to the caller.
//
// Contact records lie in the order the last evaluation's atomics gave them.
// The contact downloads report particle pairs first, then wall contacts, each
// by (id of P, id of I or the caller's wall index): two stable radix sorts (by
// I's id, then by the wall flag and P's id) order the record indices, and one
// kernel writes the caller's arrays from the records. The host sorted the
// 264-byte records themselves before, in both downloads of an output: contacts,
// geometry and forces of a drum of 50,000 (85,000 records) took 44 ms.
#pragma once
#include <cub/device/device_radix_sort.cuh>

#include "dem_kernels.cuh"

namespace dem {

// order-preserving bits of a signed integer
__device__ __forceinline__ unsigned order_bits(int v) { return (unsigned)v ^ 0x80000000u; }

__device__ __forceinline__ int reported_i(const ContactRecord& r, const int* wall_caller)
{
    return r.is_wall ? wall_caller[r.id_i] : r.id_i;
}

__global__ void __launch_bounds__(256) k_record_keys_i(const ContactRecord* rec, unsigned n, const int* wall_caller,
                                                       unsigned* key, int* idx)
{
    const unsigned r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    key[r] = order_bits(reported_i(rec[r], wall_caller));
    idx[r] = (int)r;
}

__global__ void __launch_bounds__(256) k_record_keys_p(const ContactRecord* rec, unsigned n, const int* idx,
                                                       unsigned long long* key)
{
    const unsigned k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const ContactRecord& r = rec[idx[k]];
    key[k] = ((unsigned long long)(r.is_wall ? 1u : 0u) << 32) | order_bits(r.id_p);
}

// The arrays of dem_contacts_soa and of the contact geometry; those a caller
// does not ask for are null.
struct RecordArrays {
    int *id_p, *id_i, *is_wall, *periodic;
    double *springs, *force, *overlap;             // 9, 3, 1 per record
    double *contact_point, *normal, *tangential;   // 3 each
};

__host__ __device__ __forceinline__ void put_record(const RecordArrays& a, size_t k, const ContactRecord& r, int id_i)
{
    if (a.id_p) a.id_p[k] = r.id_p;
    if (a.id_i) a.id_i[k] = id_i;
    if (a.is_wall) a.is_wall[k] = r.is_wall;
    if (a.periodic) a.periodic[k] = r.periodic;
    if (a.overlap) a.overlap[k] = r.overlap;
    if (a.springs)
        for (int c = 0; c < 9; ++c) a.springs[9 * k + c] = r.springs[c];
    for (int c = 0; c < 3; ++c) {
        if (a.force) a.force[3 * k + c] = r.force[c];
        if (a.contact_point) a.contact_point[3 * k + c] = r.contact_point[c];
        if (a.normal) a.normal[3 * k + c] = r.normal[c];
        if (a.tangential) a.tangential[3 * k + c] = r.tangential[c];
    }
}

__global__ void __launch_bounds__(256) k_record_arrays(const ContactRecord* rec, unsigned n, const int* order,
                                                       const int* wall_caller, RecordArrays a)
{
    const unsigned k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const ContactRecord& r = rec[order[k]];
    put_record(a, k, r, reported_i(r, wall_caller));
}

// forces and torques (engine order) -> caller order
__global__ void __launch_bounds__(256) k_unpack_forces(DevPtrs d, int b, double* force, double* torque)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= d.n) return;
    const size_t i = (size_t)d.caller[b][s];
    for (int c = 0; c < 3; ++c) {
        force[3 * i + c] = d.force[3 * (size_t)s + c];
        torque[3 * i + c] = d.torque[3 * (size_t)s + c];
    }
}

// list entries of the neighbour rows, and the contact records by kind (counts)
__global__ void __launch_bounds__(256) k_count(DevPtrs d, unsigned n_records, unsigned long long* out)
{
    unsigned long long v[3] = {0ull, 0ull, 0ull};
    const unsigned stride = gridDim.x * blockDim.x, t = blockIdx.x * blockDim.x + threadIdx.x;
    for (unsigned i = t; i < (unsigned)d.n; i += stride) v[0] += (unsigned long long)d.cnt[i];
    for (unsigned r = t; r < n_records; r += stride) ++v[d.records[r].is_wall ? 2 : 1];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
        if ((threadIdx.x & 31) == 0 && v[k]) atomicAdd(out + k, v[k]);
    }
}

} // namespace dem
