// hostmesh.cu — a host caller's mesh arrays, put in the kernels' layout on the device.
//
// The drop-in routines get inpoel(3,nelem), 1-based, and dNx/dNy(3,nelem) with every call.  The
// element table with its range check, the elements around each point (pointNeighbor.f90:5-43)
// and the six geometry planes are formed here from the raw arrays: at 262,144 nodes 5.4 ms of
// the call's 9.3 ms when the host formed them, ~0.1 ms on the device.
#include "cfd_kernels.cuh"

namespace cfd {

// inpoel -> int4 0-based (w = e); flags[0] = the first element with a node outside 1..npoin
// (its int4 is all zeros then, so that what reads the table stays inside the arrays).  With deg:
// deg[p] += 1 for each slot of p, rank[slot] = the count before it.  The rank depends on the
// order of the atomics; k_esup_sort removes that.
__global__ void k_elem_table(int nelem, int npoin, const int* __restrict__ inpoel,
                             int4* __restrict__ elem, int* __restrict__ deg,
                             int* __restrict__ rank, unsigned* __restrict__ flags) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nelem) return;
    int n[3];
    bool ok = true;
    for (int i = 0; i < 3; ++i) {
        n[i] = inpoel[3 * (size_t)e + i] - 1;
        ok = ok && (unsigned)n[i] < (unsigned)npoin;
    }
    if (!ok) {
        atomicMin(&flags[0], (unsigned)e);
        elem[e] = make_int4(0, 0, 0, e);
        return;
    }
    elem[e] = make_int4(n[0], n[1], n[2], e);
    if (deg)
        for (int i = 0; i < 3; ++i) rank[3 * (size_t)e + i] = atomicAdd(&deg[n[i]], 1);
}

// Exclusive prefix sums of deg in two launches: each block's sum of its kScanItems degrees (and
// the largest degree, kept complemented in flags[1]), then every block adds up the sums before
// it and scans its own.
constexpr int kScanTB = 512, kScanPer = 8, kScanItems = kScanTB * kScanPer;
__device__ __forceinline__ int block_exclusive(int v, int* warp_sums, int* total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int x = v;
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[w] = x;
    __syncthreads();
    int before = 0, all = 0;
    for (int k = 0; k < kScanTB / 32; ++k) {
        const int s = warp_sums[k];
        if (k < w) before += s;
        all += s;
    }
    __syncthreads();
    *total = all;
    return before + x - v;
}
__global__ void __launch_bounds__(kScanTB)
k_esup_sums(int npoin, const int* __restrict__ deg, int* __restrict__ sums,
            unsigned* __restrict__ flags) {
    __shared__ int ws[kScanTB / 32];
    const long b = (long)blockIdx.x * kScanItems;
    int s = 0, mx = 0;
    for (int k = 0; k < kScanPer; ++k) {
        const long i = b + k * kScanTB + threadIdx.x;
        const int d = i < npoin ? deg[i] : 0;
        s += d;
        mx = max(mx, d);
    }
    int total;
    block_exclusive(s, ws, &total);
    mx = __reduce_max_sync(0xffffffffu, mx);
    if ((threadIdx.x & 31) == 0) atomicMin(&flags[1], ~(unsigned)mx);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}
__global__ void __launch_bounds__(kScanTB)
k_esup_scan(int npoin, const int* __restrict__ deg, const int* __restrict__ sums,
            int* __restrict__ ptr) {
    __shared__ int ws[kScanTB / 32];
    int s = 0, base;
    for (int k = threadIdx.x; k < (int)blockIdx.x; k += kScanTB) s += sums[k];
    block_exclusive(s, ws, &base);
    const long b = (long)blockIdx.x * kScanItems + (long)threadIdx.x * kScanPer;
    int d[kScanPer], mine = 0;
    for (int k = 0; k < kScanPer; ++k) {
        d[k] = b + k < npoin ? deg[b + k] : 0;
        mine += d[k];
    }
    int total;
    int at = base + block_exclusive(mine, ws, &total);
    for (int k = 0; k < kScanPer; ++k)
        if (b + k < npoin) {
            ptr[b + k] = at;
            at += d[k];
            if (b + k == npoin - 1) ptr[npoin] = at;
        }
}

__global__ void k_esup_fill(int nelem, const int4* __restrict__ elem, const int* __restrict__ ptr,
                            const int* __restrict__ rank, int* __restrict__ slot,
                            const unsigned* __restrict__ flags) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nelem || flags[0] != ~0u) return;  // a bad element has no rank
    const int4 n = elem[e];
    const int nn[3] = {n.x, n.y, n.z};
    for (int i = 0; i < 3; ++i) slot[ptr[nn[i]] + rank[3 * (size_t)e + i]] = 3 * e + i;
}

// Each node's slots in ascending order, which is the reference's element order: insertion
// sort by the node's thread (six slots on a triangle mesh).  Nodes of more than
// kEsupSortMax slots are left alone; their caller forms the lists on the host.
__global__ void k_esup_sort(int npoin, const int* __restrict__ ptr, int* __restrict__ slot,
                            const unsigned* __restrict__ flags) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= npoin || flags[0] != ~0u) return;
    const int b = ptr[p], n = ptr[p + 1] - b;
    if (n > kEsupSortMax) return;
    for (int i = 1; i < n; ++i) {
        const int v = slot[b + i];
        int j = i;
        for (; j > 0 && slot[b + j - 1] > v; --j) slot[b + j] = slot[b + j - 1];
        slot[b + j] = v;
    }
}

// dNx(3,nelem), dNy(3,nelem) <-> the six planes [dNx1|dNx2|dNx3|dNy1|dNy2|dNy3], elements
// [e0, e1) of nelem
__global__ void k_geo_planes(int e0, int e1, int nelem, const double* __restrict__ dnx,
                             const double* __restrict__ dny, double* __restrict__ geo) {
    const int e = e0 + blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= e1) return;
    for (int i = 0; i < 3; ++i) {
        geo[i * (size_t)nelem + e] = dnx[3 * (size_t)e + i];
        geo[(3 + i) * (size_t)nelem + e] = dny[3 * (size_t)e + i];
    }
}
__global__ void k_geo_rows(int nelem, const double* __restrict__ geo, double* __restrict__ dnx,
                           double* __restrict__ dny) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nelem) return;
    for (int i = 0; i < 3; ++i) {
        dnx[3 * (size_t)e + i] = geo[i * (size_t)nelem + e];
        dny[3 * (size_t)e + i] = geo[(3 + i) * (size_t)nelem + e];
    }
}

// a 1-based index list -> 0-based; flag = the first entry outside 1..npoin (written as 0)
__global__ void k_index_list(int n, int npoin, const int* __restrict__ in, int* __restrict__ out,
                             unsigned* __restrict__ flag) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int v = in[k] - 1;
    const bool ok = (unsigned)v < (unsigned)npoin;
    if (!ok) atomicMin(flag, (unsigned)k);
    out[k] = ok ? v : 0;
}

long esup_scan_blocks(long npoin) { return (npoin + kScanItems - 1) / kScanItems; }

cudaError_t launch_elem_table(cudaStream_t st, int nelem, int npoin, const int* inpoel, int4* elem,
                              int* deg, int* rank, unsigned* flags) {
    k_elem_table<<<blocks_for(nelem, 256), 256, 0, st>>>(nelem, npoin, inpoel, elem, deg, rank, flags);
    g_launches.fetch_add(1, std::memory_order_relaxed);
    return cudaGetLastError();
}

cudaError_t launch_esup(cudaStream_t st, int nelem, int npoin, const int4* elem, const int* deg,
                        const int* rank, int* sums, int* ptr, int* slot, unsigned* flags) {
    const unsigned nb = (unsigned)esup_scan_blocks(npoin);
    k_esup_sums<<<nb, kScanTB, 0, st>>>(npoin, deg, sums, flags);
    k_esup_scan<<<nb, kScanTB, 0, st>>>(npoin, deg, sums, ptr);
    k_esup_fill<<<blocks_for(nelem, 256), 256, 0, st>>>(nelem, elem, ptr, rank, slot, flags);
    k_esup_sort<<<blocks_for(npoin, 256), 256, 0, st>>>(npoin, ptr, slot, flags);
    g_launches.fetch_add(4, std::memory_order_relaxed);
    return cudaGetLastError();
}

}  // namespace cfd
