// Re-sort of the particles by cell and transfers between original order (one
// row of components per particle) and storage order (an array per component),
// for one simulation (arguments by value) or for many in one launch (a device
// table of arguments, member = blockIdx.x).
//
// Both are streams of a few arrays per particle, so bytes and, for small
// simulations, launches bound them: a re-sort moves every array of a particle
// in one kernel that reads the permutation once (as a kernel per array it was
// 27 launches a re-sort), and a transfer takes the components that keep
// original order (zero through every step) along in the same kernel (they were
// strided 4-byte-row copies: 3 ms a field of 16.8M particles).
#include <cuda_runtime.h>

#include <algorithm>

#include "mpm_device.cuh"
#include "mpm_kernels.h"

namespace mpm {

namespace {

constexpr int XFER_THREADS = 256;
constexpr int XFER_CHUNK = 4 * XFER_THREADS;   // elements of a job per block

// Run f(job, i) for every element i < n(job): one job by value, or a table.
template <class J, class N, class F>
__device__ __forceinline__ void for_one(const J& j, N&& n, F&& f) {
    const int i = blockIdx.x * XFER_THREADS + threadIdx.x;
    if (i < n(j)) f(j, i);
}
template <class J, class N, class F>
__device__ __forceinline__ void for_many(const J* __restrict__ jobs, N&& n, F&& f) {
    const J& j = jobs[blockIdx.x];
    const int total = n(j);
    for (int c = blockIdx.y; (long long)c * XFER_CHUNK < total; c += gridDim.y) {
        #pragma unroll 1
        for (int k = 0; k < XFER_CHUNK; k += XFER_THREADS) {
            const int i = c * XFER_CHUNK + k + (int)threadIdx.x;
            if (i < total) f(j, i);
        }
    }
}
inline dim3 many_grid(int njobs, int most) {
    return dim3(njobs, std::min(65535, std::max(1, (most + XFER_CHUNK - 1) / XFER_CHUNK)));
}
inline int one_grid(int n) { return (n + XFER_THREADS - 1) / XFER_THREADS; }

// ---------------------------------------------------------------------------
// Re-sort: key = current cell (ncell for a particle outside the mesh), counting
// sort whose ranks come from the counting atomics, then each bucket sorted by
// storage index, so the result is the stable order whatever order the atomics
// took.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void sort_clear(const SortJob& J, int c) {
    J.count[c] = 0;
    if (c < J.nx * J.ny) J.cflag[c] = 0;
}
__device__ __forceinline__ void sort_key(const SortJob& J, int q) {
    const int i = locate_axis(J.x[q], J.hx, J.nx);
    const int j = locate_axis(J.y[q], J.hy, J.ny);
    int k;
    if (i < 0 || i >= J.nx || j < 0 || j >= J.ny) {
        k = J.nx * J.ny;
        atomicOr(&J.ctl->status, ST_OUT_OF_MESH);
    } else {
        k = j * J.nx + i;
    }
    J.key[q] = k;
    J.rank[q] = atomicAdd(&J.count[k], 1);
}
__device__ __forceinline__ void sort_place(const SortJob& J, int q) {
    J.perm[J.start[J.key[q]] + J.rank[q]] = q;
}
// (The counts are zero between sorts: a launch less before the keys.)
__device__ __forceinline__ void sort_bucket(const SortJob& J, int c) {
    sort_clear(J, c);
    const int b = J.start[c], e = J.start[c + 1];
    int* __restrict__ perm = J.perm;
    #pragma unroll 1
    for (int i = b + 1; i < e; ++i) {
        const int v = perm[i];
        int j = i - 1;
        #pragma unroll 1
        while (j >= b && perm[j] > v) {
            perm[j + 1] = perm[j];
            --j;
        }
        perm[j + 1] = v;
    }
}
// Every array of the particle at storage slot i after the sort.
__device__ __forceinline__ void sort_move(const SortJob& J, int i) {
    const int p = J.perm[i];
    constexpr int G = 6;   // loads in flight before their stores
    #pragma unroll 1
    for (int f0 = 0; f0 < J.nf; f0 += G) {
        uint32_t v[G];
        #pragma unroll
        for (int f = 0; f < G; ++f)
            if (f0 + f < J.nf) v[f] = J.src[f0 + f][p];
        #pragma unroll
        for (int f = 0; f < G; ++f)
            if (f0 + f < J.nf) J.dst[f0 + f][i] = v[f];
    }
    J.mat_dst[i] = J.mat_src[p];
    if (J.pvc_src) J.pvc_dst[i] = J.pvc_src[p];
    if (J.trfn_src) {
        J.trfn_dst[i] = J.trfn_src[p];
        J.trtau_dst[i] = J.trtau_src[p];
    }
}

struct Particles_ { __device__ int operator()(const SortJob& J) const { return J.np; } };
struct Buckets_ { __device__ int operator()(const SortJob& J) const { return J.nx * J.ny + 1; } };

__global__ void __launch_bounds__(XFER_THREADS) k_sort_clear(const __grid_constant__ SortJob J) {
    for_one(J, Buckets_{}, [](const SortJob& j, int i) { sort_clear(j, i); });
}
#define MPM_SORT_KERNELS(name, count_of, fn)                                                              \
    __global__ void __launch_bounds__(XFER_THREADS) name(const __grid_constant__ SortJob J) {             \
        for_one(J, count_of{}, [](const SortJob& j, int i) { fn(j, i); });                                \
    }                                                                                                     \
    __global__ void __launch_bounds__(XFER_THREADS) name##_many(const SortJob* __restrict__ jobs) {       \
        for_many(jobs, count_of{}, [](const SortJob& j, int i) { fn(j, i); });                            \
    }
MPM_SORT_KERNELS(k_sort_keys, Particles_, sort_key)
MPM_SORT_KERNELS(k_sort_place, Particles_, sort_place)
MPM_SORT_KERNELS(k_sort_buckets, Buckets_, sort_bucket)
MPM_SORT_KERNELS(k_sort_move, Particles_, sort_move)
#undef MPM_SORT_KERNELS

__global__ void k_scan_blocks(const int* __restrict__ in, int* __restrict__ out, int n,
                              int* __restrict__ block_sums) {
    const int i = blockIdx.x * 1024 + threadIdx.x;
    const int v = i < n ? in[i] : 0;
    int total;
    const int ex = block_exclusive_scan(v, &total);
    if (i < n) out[i] = ex;
    if (threadIdx.x == 0) block_sums[blockIdx.x] = total;
}

__global__ void k_scan_sums(int* __restrict__ block_sums, int nb) {
    __shared__ int carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int base = 0; base < nb; base += 1024) {
        const int i = base + threadIdx.x;
        const int v = i < nb ? block_sums[i] : 0;
        int total;
        const int ex = block_exclusive_scan(v, &total);
        if (i < nb) block_sums[i] = ex + carry;
        __syncthreads();
        if (threadIdx.x == 0) carry += total;
        __syncthreads();
    }
    if (threadIdx.x == 0) block_sums[nb] = carry;
}

__global__ void k_scan_add(int* __restrict__ out, int n, const int* __restrict__ block_sums) {
    const int i = blockIdx.x * 1024 + threadIdx.x;
    if (i < n) out[i] += block_sums[blockIdx.x];
    if (i == n) out[n] = block_sums[gridDim.x];   // grand total
}

// Chunk c of a job's counts by one CTA, start[n] with the last one: every CTA
// adds up the counts before its chunk itself, so that one launch scans them all
// (up to SORT_MANY_CELLS: the last chunk reads 1 MB of L2).  Bound by the two
// round trips of loading and storing; 16-byte accesses, the loads of a thread's
// four pieces in flight together (21k cells: 14.4 us by one CTA 8 counts a
// thread and round, 3.5 so; a three-launch scan takes 8).
constexpr int SCAN_PIECES = 4, SCAN_CHUNK = SCAN_PIECES * 4 * 1024;
__device__ __forceinline__ void sort_scan(const SortJob& J, int c) {
    const int n = J.nx * J.ny + 1, t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int base = c * SCAN_CHUNK;
    if (base >= n) return;
    __shared__ __align__(16) int s_part[SCAN_PIECES * 32];   // (also read and written four at a time)
    __shared__ int s_before[32], s_carry;
    const int4* __restrict__ in = reinterpret_cast<const int4*>(J.count);
    int4 v[SCAN_PIECES];
    #pragma unroll
    for (int r = 0; r < SCAN_PIECES; ++r) {
        const int i = base + 4 * (r * 1024 + t);
        v[r] = make_int4(0, 0, 0, 0);
        if (i + 4 <= n) {
            v[r] = in[i >> 2];
        } else {
            if (i < n) v[r].x = J.count[i];
            if (i + 1 < n) v[r].y = J.count[i + 1];
            if (i + 2 < n) v[r].z = J.count[i + 2];
        }
    }
    int before = 0;
    #pragma unroll 8
    for (int i = t; i < base / 4; i += 1024) {
        const int4 w = in[i];
        before += w.x + w.y + w.z + w.w;
    }
    before = __reduce_add_sync(0xffffffffu, before);
    if (lane == 0) s_before[warp] = before;
    int at[SCAN_PIECES];
    #pragma unroll
    for (int r = 0; r < SCAN_PIECES; ++r) {
        const int own = v[r].x + v[r].y + v[r].z + v[r].w;
        at[r] = own;
        #pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, at[r], o);
            if (lane >= o) at[r] += u;
        }
        if (lane == 31) s_part[r * 32 + warp] = at[r];
        at[r] -= own;
    }
    __syncthreads();
    if (warp == 0) {   // the warps' sums, piece after piece
        int4 q = reinterpret_cast<const int4*>(s_part)[lane];
        const int own = q.x + q.y + q.z + q.w;
        int u = own;
        #pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int w = __shfl_up_sync(0xffffffffu, u, o);
            if (lane >= o) u += w;
        }
        u += __reduce_add_sync(0xffffffffu, s_before[lane]);
        if (lane == 31) s_carry = u;
        u -= own;
        q = make_int4(u, u + q.x, u + q.x + q.y, u + q.x + q.y + q.z);
        reinterpret_cast<int4*>(s_part)[lane] = q;
    }
    __syncthreads();
    #pragma unroll
    for (int r = 0; r < SCAN_PIECES; ++r) {
        const int i = base + 4 * (r * 1024 + t);
        const int a = at[r] + s_part[r * 32 + warp];
        const int4 q = make_int4(a, a + v[r].x, a + v[r].x + v[r].y, a + v[r].x + v[r].y + v[r].z);
        if (i + 4 <= n) {
            reinterpret_cast<int4*>(J.start)[i >> 2] = q;
        } else {
            if (i < n) J.start[i] = q.x;
            if (i + 1 < n) J.start[i + 1] = q.y;
            if (i + 2 < n) J.start[i + 2] = q.z;
        }
    }
    if (t == 0 && n - base <= SCAN_CHUNK) J.start[n] = s_carry;
}
__global__ void __launch_bounds__(1024) k_sort_scan(const __grid_constant__ SortJob J) { sort_scan(J, blockIdx.x); }
__global__ void __launch_bounds__(1024) k_sort_scan_many(const SortJob* __restrict__ jobs) {
    sort_scan(jobs[blockIdx.x], blockIdx.y);
}

__global__ void k_put_descs(const DescPut* __restrict__ puts, int n) {
    for (int i = blockIdx.x; i < n; i += gridDim.x) {
        const int* a = reinterpret_cast<const int*>(&puts[i].S);
        int* b = reinterpret_cast<int*>(puts[i].dst);
        for (int w = threadIdx.x; w < (int)(sizeof(SimDev) / 4); w += blockDim.x) b[w] = a[w];
    }
}

// ---------------------------------------------------------------------------
// Field transfers
// ---------------------------------------------------------------------------
struct Mapped_ { __device__ int operator()(const FieldMap& F) const { return F.np; } };

// (all loads of a round in flight before its stores)
constexpr int FIELD_G = 6;
__device__ __forceinline__ void field_in(const FieldMap& F, int i) {
    const size_t o = F.pid ? F.pid[i] : i;
    #pragma unroll 1
    for (int c0 = 0; c0 < F.ncomp; c0 += FIELD_G) {
        float v[FIELD_G];
        #pragma unroll
        for (int c = 0; c < FIELD_G; ++c)
            v[c] = c0 + c < F.ncomp && F.aos ? F.aos[o * F.ncomp + c0 + c] : 0.0f;
        #pragma unroll
        for (int c = 0; c < FIELD_G; ++c) {
            if (c0 + c >= F.ncomp) continue;
            if (F.comp[c0 + c]) F.comp[c0 + c][i] = v[c];
            else if (F.slot[c0 + c] >= 0) F.passive[o * PASSIVE_N + F.slot[c0 + c]] = v[c];
        }
    }
}
__device__ __forceinline__ void field_out(const FieldMap& F, int i) {
    const size_t o = F.pid ? F.pid[i] : i;
    #pragma unroll 1
    for (int c0 = 0; c0 < F.ncomp; c0 += FIELD_G) {
        float v[FIELD_G];
        #pragma unroll
        for (int c = 0; c < FIELD_G; ++c) {
            v[c] = 0.0f;
            if (c0 + c >= F.ncomp) continue;
            if (F.comp[c0 + c]) v[c] = F.comp[c0 + c][i];
            else if (F.slot[c0 + c] >= 0) v[c] = F.passive[o * PASSIVE_N + F.slot[c0 + c]];
        }
        #pragma unroll
        for (int c = 0; c < FIELD_G; ++c)
            if (c0 + c < F.ncomp) F.aos[o * F.ncomp + c0 + c] = v[c];
    }
}
template <bool IN>
__global__ void __launch_bounds__(XFER_THREADS) k_field(const __grid_constant__ FieldMap F) {
    for_one(F, Mapped_{}, [](const FieldMap& f, int i) {
        if (IN) field_in(f, i);
        else field_out(f, i);
    });
}
template <bool IN>
__global__ void __launch_bounds__(XFER_THREADS) k_field_many(const FieldMap* __restrict__ maps) {
    for_many(maps, Mapped_{}, [](const FieldMap& f, int i) {
        if (IN) field_in(f, i);
        else field_out(f, i);
    });
}

template <class T>
__global__ void k_gather(const T* __restrict__ src, T* __restrict__ dst, const int* __restrict__ perm, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = src[perm[i]];
}

}  // namespace

cudaError_t launch_gather_pairs(const uint16_t* src, uint16_t* dst, const int* perm, int n, cudaStream_t s) {
    if (n > 0) k_gather<<<one_grid(n), XFER_THREADS, 0, s>>>(src, dst, perm, n);
    return cudaGetLastError();
}
cudaError_t launch_gather_pairs(const float2* src, float2* dst, const int* perm, int n, cudaStream_t s) {
    if (n > 0) k_gather<<<one_grid(n), XFER_THREADS, 0, s>>>(src, dst, perm, n);
    return cudaGetLastError();
}

cudaError_t launch_sort_order(const SortJob& J, int* block_sums, bool buckets, cudaStream_t s) {
    const int nb = J.nx * J.ny + 1, n = (nb + 1024) / 1024;   // room for start[nb]
    if (!buckets) k_sort_clear<<<one_grid(nb), XFER_THREADS, 0, s>>>(J);
    if (J.np > 0) k_sort_keys<<<one_grid(J.np), XFER_THREADS, 0, s>>>(J);
    if (nb - 1 <= SORT_MANY_CELLS) {
        k_sort_scan<<<(nb + SCAN_CHUNK - 1) / SCAN_CHUNK, 1024, 0, s>>>(J);
    } else {
        k_scan_blocks<<<n, 1024, 0, s>>>(J.count, J.start, nb, block_sums);
        k_scan_sums<<<1, 1024, 0, s>>>(block_sums, n);
        k_scan_add<<<n, 1024, 0, s>>>(J.start, nb, block_sums);
    }
    if (J.np > 0) k_sort_place<<<one_grid(J.np), XFER_THREADS, 0, s>>>(J);
    if (buckets) k_sort_buckets<<<one_grid(nb), XFER_THREADS, 0, s>>>(J);
    return cudaGetLastError();
}

cudaError_t launch_sort_move(const SortJob& J, cudaStream_t s) {
    if (J.np > 0) k_sort_move<<<one_grid(J.np), XFER_THREADS, 0, s>>>(J);
    return cudaGetLastError();
}

cudaError_t launch_sort_many(const SortJob* jobs, int n, int most_np, int most_cells, cudaStream_t s) {
    if (n < 1) return cudaSuccess;
    const dim3 gp = many_grid(n, most_np), gc = many_grid(n, most_cells + 1);
    k_sort_keys_many<<<gp, XFER_THREADS, 0, s>>>(jobs);
    k_sort_scan_many<<<dim3(n, (most_cells + SCAN_CHUNK) / SCAN_CHUNK), 1024, 0, s>>>(jobs);
    k_sort_place_many<<<gp, XFER_THREADS, 0, s>>>(jobs);
    k_sort_buckets_many<<<gc, XFER_THREADS, 0, s>>>(jobs);
    k_sort_move_many<<<gp, XFER_THREADS, 0, s>>>(jobs);
    return cudaGetLastError();
}

cudaError_t launch_put_descs(const DescPut* puts, int n, cudaStream_t s) {
    if (n > 0) k_put_descs<<<std::min(n, 1024), 128, 0, s>>>(puts, n);
    return cudaGetLastError();
}

cudaError_t launch_field(const FieldMap& F, bool in, cudaStream_t s) {
    if (F.np > 0) {
        if (in) k_field<true><<<one_grid(F.np), XFER_THREADS, 0, s>>>(F);
        else k_field<false><<<one_grid(F.np), XFER_THREADS, 0, s>>>(F);
    }
    return cudaGetLastError();
}

cudaError_t launch_field_many(const FieldMap* maps, int n, int most_np, bool in, cudaStream_t s) {
    if (n > 0 && most_np > 0) {
        const dim3 g = many_grid(n, most_np);
        if (in) k_field_many<true><<<g, XFER_THREADS, 0, s>>>(maps);
        else k_field_many<false><<<g, XFER_THREADS, 0, s>>>(maps);
    }
    return cudaGetLastError();
}

}  // namespace mpm
