// gg_points.cu -- material point → element mapping on sm_100a.
//
//  k_locate        bit-exact Mesh_RegularAlgorithms_SearchElements
//                  (StgDomain/Mesh/src/Mesh_RegularAlgorithms.cxx:191-224) + per-element
//                  histogram; the count a point finds is its place in the element
//  k_scan_*        exclusive scan of the histogram → CSR offsets
//  k_scatter       counting-sort scatter by offset + place (arbitrary order inside an element)
//  k_segsort       per-element sort by input index, which restores the order that
//                  _CoincidentMapper_Map (PICellerator/MaterialPoints/src/
//                  CoincidentMapper.cxx:190-215) rebuilds: increasing point index
//  k_gather_points ξ (closed form of the Newton step of ElementType.cxx:221-338 on an
//                  axis-aligned element), material, plastic strain in sorted order
//
// All integer work; HBM-bound.  Every kernel is grid-stride and sized from the SM count.
#include "gg_internal.cuh"
#include "gg_kernels.cuh"

namespace gg {

// place != null: place[p] = the point's place among its element's points (arrival order).
// place == null: the place is kept in cell[p] itself, above the kCellBits of the element
// (kPlaceMax where it does not fit), and k_scatter takes it out again.  Counting once, here,
// instead of a second time in k_scatter, halves the random atomics, which with the random
// stores of the scatter are what the sort of a shuffled swarm costs (28.3 M points on 2^20
// elements: this kernel 370 µs with the atomics returning, 250 without, but k_scatter's own
// count cost as much again; the whole location 1.26 → 0.85 ms with the steps below).
__global__ void k_locate(MeshK mk, int64_t np, const double* __restrict__ x,
                         uint32_t* __restrict__ cell, int32_t* __restrict__ count,
                         int32_t* __restrict__ flag, int32_t* __restrict__ place) {
    const int dim = mk.dim;
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < np;
         p += (int64_t)gridDim.x * blockDim.x) {
        int inds[3] = {0, 0, 0};
        bool inside = true;
        for (int d = 0; d < dim; d++) {
            const double v = x[p * dim + d];
            const double dmax = __dsub_rn(v, mk.max[d]);
            if (dmax >= -1e-12 && dmax <= 1e-12) {          // Num_Approx(x - max, 0)
                inds[d] = mk.n[d] - 1;
            } else if (v < mk.min[d] || v > mk.max[d]) {
                inside = false;
            } else {
                const double out = __ddiv_rn(__dsub_rn(v, mk.min[d]), mk.sep[d]);
                const double ip = trunc(out);               // modf: integral part
                const double frac = __dsub_rn(out, ip);     // exact fractional part
                int i = (int)ip;
                if (i > 0 && frac >= -1e-12 && frac <= 1e-12) i--;  // lower element wins
                if (i >= mk.n[d]) i = mk.n[d] - 1;
                inds[d] = i;
            }
        }
        if (inside) {
            const int64_t e = inds[0] + (int64_t)mk.n[0] * (inds[1] + (int64_t)mk.n[1] * inds[2]);
            const int32_t at = atomicAdd(&count[e], 1);
            if (place) {
                cell[p] = (uint32_t)e;
                place[p] = at;
            } else {
                cell[p] = (uint32_t)e | (uint32_t)(at < kPlaceMax ? at : kPlaceMax) << kCellBits;
            }
        } else {
            cell[p] = (uint32_t)mk.nel;
            atomicAdd(flag, 1);
        }
    }
}

// ---- exclusive scan, 3 phases (1024 items per block) -------------------------------
__global__ void k_scan_blocks(const int32_t* __restrict__ in, int64_t n, int32_t* __restrict__ out,
                              int32_t* __restrict__ block_sums) {
    __shared__ int32_t warp_tot[32];
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int32_t v = i < n ? in[i] : 0;
    int32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) warp_tot[wid] = incl;
    __syncthreads();
    if (wid == 0) {
        int32_t w = lane < (int)(blockDim.x >> 5) ? warp_tot[lane] : 0;
        int32_t wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int32_t t = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += t;
        }
        warp_tot[lane] = wi - w;  // exclusive prefix of warp totals
        if (lane == 31) block_sums[blockIdx.x] = wi;
    }
    __syncthreads();
    if (i < n) out[i] = incl - v + warp_tot[wid];
}

__global__ void k_scan_sums(int32_t* __restrict__ sums, int64_t nblocks, int32_t* __restrict__ total) {
    // one block: sequential carry over chunks of blockDim
    __shared__ int32_t warp_tot[32];
    __shared__ int32_t carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int64_t base = 0; base < nblocks; base += blockDim.x) {
        const int64_t i = base + threadIdx.x;
        int32_t v = i < nblocks ? sums[i] : 0;
        int32_t incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int32_t t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        if (lane == 31) warp_tot[wid] = incl;
        __syncthreads();
        if (wid == 0) {
            int32_t w = lane < (int)(blockDim.x >> 5) ? warp_tot[lane] : 0;
            int32_t wi = w;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                int32_t t = __shfl_up_sync(0xffffffffu, wi, o);
                if (lane >= o) wi += t;
            }
            warp_tot[lane] = wi - w;
        }
        __syncthreads();
        const int32_t c = carry;
        if (i < nblocks) sums[i] = c + incl - v + warp_tot[wid];
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) carry = c + incl + warp_tot[wid];
        __syncthreads();
    }
    if (threadIdx.x == 0) *total = carry;
}

__global__ void k_scan_add(int32_t* __restrict__ out, int64_t n, const int32_t* __restrict__ sums,
                           const int32_t* __restrict__ total) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) out[i] += sums[blockIdx.x];
    if (i == 0) out[n] = *total;
}

// unsorted[offset + place] = p for the points of elements e_lo … e_hi − 1.  keep: the places in
// cell stay for another window (place == null).  The stores are single words all over the
// window; while it stays in L2 its sectors fill up there, beyond that they go to memory one
// word at a time, so the host splits the elements into windows (launch_scatter).
__global__ void k_scatter(int64_t np, uint32_t e_lo, uint32_t e_hi, int keep, uint32_t* __restrict__ cell,
                          const int32_t* __restrict__ offsets, const int32_t* __restrict__ place,
                          int32_t* __restrict__ unsorted) {
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < np;
         p += (int64_t)gridDim.x * blockDim.x) {
        uint32_t e = __ldcs(cell + p);
        int32_t at;
        if (place) {
            if (e < e_lo || e >= e_hi) continue;
            at = __ldcs(place + p);
        } else {
            at = (int32_t)(e >> kCellBits);
            e &= (1u << kCellBits) - 1u;
            if (!keep) __stcs(cell + p, e);
            if (e < e_lo || e >= e_hi || at >= kPlaceMax) continue;  // kPlaceMax: the element is refused
        }
        unsorted[offsets[e] + at] = (int32_t)p;
    }
}

void launch_scatter(int64_t np, int64_t nel, uint32_t* cell, const int32_t* offsets, const int32_t* place,
                    int32_t* unsorted, cudaStream_t st) {
    // 28.3 M points in windows of 16 / 32 / 64 / 128 MB: the whole location 1.03 / 0.89 / 0.85 /
    // 1.07 ms (a window costs another read of the cells, 128 MB no longer stays in L2)
    constexpr int64_t words = (int64_t(64) << 20) / 4;
    const int64_t passes = (np + words - 1) / words;
    for (int64_t w = 0; w < passes; w++)
        k_scatter<<<grid_for(np, 256), 256, 0, st>>>(np, (uint32_t)(nel * w / passes), (uint32_t)(nel * (w + 1) / passes),
                                                     w + 1 < passes, cell, offsets, place, unsorted);
}

// Batcher's odd-even merge sort of K values in registers, ascending.
template <int K>
__device__ __forceinline__ void sort_registers(int32_t (&v)[K]) {
    constexpr int L = K == 16 ? 4 : K == 32 ? 5 : 6;
#pragma unroll
    for (int lp = 0; lp < L; lp++)
#pragma unroll
        for (int lk = lp; lk >= 0; lk--)
#pragma unroll
            for (int i = 0; i < K; i++) {
                const int p = 1 << lp, k = 1 << lk, j0 = k % p;
                if (i >= j0 && (i - j0) % (2 * k) < k && i + k < K && i / (2 * p) == (i + k) / (2 * p)) {
                    const int32_t lo = min(v[i], v[i + k]), hi = max(v[i], v[i + k]);
                    v[i] = lo;
                    v[i + k] = hi;
                }
            }
}

template <int K>
__device__ __forceinline__ void sort_segment(int32_t* seg, int n) {
    int32_t v[K];
#pragma unroll
    for (int j = 0; j < K; j++) v[j] = j < n ? seg[j] : INT32_MAX;
    sort_registers<K>(v);
#pragma unroll
    for (int j = 0; j < K; j++)
        if (j < n) seg[j] = v[j];
}

// Every element's point indices ascending (they are distinct).  A block takes `per` elements
// (at most 128, one per thread): where each holds at most 64 points, their contiguous range
// passes through shared memory and one thread sorts each element with a network in registers,
// 191 compare-exchanges for up to 32 points.  One warp per element ranking each index against
// all others took 300 µs for 28.3 M points on 2^20 elements (issue-bound); the network needs a
// tenth of the instructions and leaves the two passes over the indices.  Blocks with a larger
// element or a range beyond kSegCap rank them, a warp per element; the ranking is
// quadratic, so a block then wants few elements (segsort_per).
// kInPlace: perm is unsorted, elements beyond kPlaceSort points are left alone and counted in
// flags[1].  Otherwise unsorted is overwritten with the sorted points' element, and flags[1]
// becomes the largest element's count.
template <bool kInPlace>
__global__ void __launch_bounds__(kSegBlock)
k_segsort(int64_t nel, int per, const int32_t* __restrict__ offsets, int32_t* unsorted, int32_t* perm, int32_t* flags) {
    __shared__ int32_t buf[kSegCap];
    __shared__ int s_most[kSegBlock / 32];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    for (int64_t e0 = (int64_t)blockIdx.x * per; e0 < nel; e0 += (int64_t)gridDim.x * per) {
        const int64_t e = e0 + threadIdx.x, e1 = e0 + per < nel ? e0 + per : nel;
        const int32_t r0 = offsets[e0], r1 = offsets[e1];
        const int32_t b = e < e1 ? offsets[e] : r1, n = e < e1 ? offsets[e + 1] - b : 0;
        const int most_w = __reduce_max_sync(0xffffffffu, n);
        if (lane == 0) s_most[wib] = most_w;
        __syncthreads();
        int most = 0;
#pragma unroll
        for (int w = 0; w < kSegBlock / 32; w++) most = max(most, s_most[w]);
        if (!kInPlace && threadIdx.x == 0) atomicMax(&flags[1], most);
        // (in a block of a few elements hardly a thread sorts: from 33 points on its warps rank faster)
        if (most <= (per < 32 ? 32 : 64) && r1 - r0 <= kSegCap) {
            for (int32_t i = r0 + threadIdx.x; i < r1; i += kSegBlock) buf[i - r0] = unsorted[i];
            __syncthreads();
            int32_t* seg = buf + (b - r0);
            if (most <= 16) sort_segment<16>(seg, n);
            else if (most <= 32) sort_segment<32>(seg, n);
            else sort_segment<64>(seg, n);
            __syncthreads();
            for (int32_t i = r0 + threadIdx.x; i < r1; i += kSegBlock) perm[i] = buf[i - r0];
            if (!kInPlace) {
                __syncthreads();
                for (int k = 0; k < n; k++) seg[k] = (int32_t)e;
                __syncthreads();
                for (int32_t i = r0 + threadIdx.x; i < r1; i += kSegBlock) unsorted[i] = buf[i - r0];
            }
        } else {
            int32_t* mine = buf + wib * kPlaceSort;
            for (int64_t q = e0 + wib; q < e1; q += kSegBlock / 32) {
                const int32_t qb = offsets[q], qn = offsets[q + 1] - qb;
                if (qn <= kPlaceSort) {
                    for (int k = lane; k < qn; k += 32) mine[k] = unsorted[qb + k];
                    __syncwarp();
                    for (int k = lane; k < qn; k += 32) {
                        const int32_t v = mine[k];
                        int rank = 0;
                        for (int j = 0; j < qn; j++) rank += (mine[j] < v);
                        perm[qb + rank] = v;
                    }
                } else if (kInPlace) {
                    if (lane == 0) atomicAdd(&flags[1], 1);
                    continue;
                } else {
                    for (int k = lane; k < qn; k += 32) {
                        const int32_t v = unsorted[qb + k];
                        int rank = 0;
                        for (int j = 0; j < qn; j++) rank += (unsorted[qb + j] < v);
                        perm[qb + rank] = v;
                    }
                }
                __syncwarp();
                if (!kInPlace)
                    for (int k = lane; k < qn; k += 32) unsorted[qb + k] = (int32_t)q;
                __syncwarp();
            }
        }
        __syncthreads();
    }
}
template __global__ void k_segsort<true>(int64_t, int, const int32_t* __restrict__, int32_t*, int32_t*, int32_t*);

// Elements per block of k_segsort.  Above 40 points on average many elements exceed what the
// network takes: one per warp (µs of a location, 128 / 4 per block: 64² of 64 120 / 74, of 300
// 871 / 160, 16² of 1000 7273 / 352); on meshes that leave the SMs idle from 32 points on (16³
// of 40 68 / 60), and always on those of up to four elements per SM.  Below, a warp's worth at least: large meshes in blocks of 128, smaller ones
// on four blocks per SM (64² of 20 in blocks of 4: 59 µs, of 32 and 128: 50).
int segsort_per(int64_t np, int64_t nel) {
    const int64_t sms = num_sms();
    if (np > 40 * nel || (np > 32 * nel && nel < 32 * sms) || nel <= 4 * sms) return kSegBlock / 32;
    int per = kSegBlock;
    while (per > 32 && nel < per * 4 * sms) per /= 2;
    return per;
}

int segsort_grid(int64_t nel, int per) {
    const int64_t g = (nel + per - 1) / per, cap = 32 * (int64_t)num_sms();
    return (int)(g < 1 ? 1 : g < cap ? g : cap);
}

// mat_in / ps_in null: zero for every point (a swarm of one material, no plastic strain), so
// that their random reads, a DRAM sector each, are left out.
__global__ void k_gather_points(MeshK mk, int64_t np_in, const int32_t* __restrict__ perm,
                                const int32_t* __restrict__ cell_s, const double2* __restrict__ axes,
                                const double* __restrict__ x, const int32_t* __restrict__ mat_in,
                                const double* __restrict__ ps_in, double* __restrict__ xi_s,
                                int32_t* __restrict__ mat_s, double* __restrict__ ps_s) {
    const int dim = mk.dim;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < np_in;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t p = perm[i];
        const uint32_t e = (uint32_t)cell_s[i];
        mat_s[i] = mat_in ? mat_in[p] : 0;
        ps_s[i] = ps_in ? ps_in[p] : 0.0;
        const uint32_t r = e / (uint32_t)mk.n[0];
        const uint32_t idx[3] = {e - r * (uint32_t)mk.n[0], r % (uint32_t)mk.n[1], r / (uint32_t)mk.n[1]};
        const double2* ax = axes;
        for (int d = 0; d < dim; d++) {
            // Newton from ξ=0 on an affine element: rhs = x − centre, J = half the width
            const double2 g = ax[idx[d]];
            xi_s[(int64_t)d * np_in + i] = __ddiv_rn(__dsub_rn(x[(int64_t)p * dim + d], g.x), g.y);
            ax += mk.n[d];
        }
    }
}

// centre and half width of every element along each axis, axis after axis: the doubles
// vert_coord_d gives, worked out once per mesh instead of three divisions per point and axis
__global__ void k_axes(MeshK mk, double2* __restrict__ axes) {
    int at = blockIdx.x * blockDim.x + threadIdx.x;
    for (int d = 0; d < mk.dim; d++) {
        if (at < mk.n[d]) {
            int base = 0;
            for (int o = 0; o < d; o++) base += mk.n[o];
            const double lo = vert_coord_d(mk, d, at), hi = vert_coord_d(mk, d, at + 1);
            axes[base + at] = make_double2(__dmul_rn(0.5, __dadd_rn(lo, hi)), __dmul_rn(0.5, __dsub_rn(hi, lo)));
            return;
        }
        at -= mk.n[d];
    }
}

const double2* element_axes(Handle& H) {
    if (!H.axes.p) {
        int n = 0;
        for (int d = 0; d < H.dim; d++) n += H.mk.n[d];
        H.axes.ensure(sizeof(double2) * n);
        k_axes<<<(n + 127) / 128, 128, 0, H.stream>>>(H.mk, H.axes.as<double2>());
        GG_CUDA(cudaGetLastError());
    }
    return H.axes.as<double2>();
}

// ------------------------------------------------------------------ host driver ----
int grid_for(int64_t n, int block) {
    int64_t g = (n + block - 1) / block;
    const int cap = num_sms() * 16;
    if (g > cap) g = cap;
    if (g < 1) g = 1;
    return (int)g;
}

// out = exclusive prefix sum of in[0..n) (device), *total_host = the sum (synchronises).
void exclusive_scan_i32(Handle& H, const int32_t* in, int32_t* out, int64_t n, DBuf& tmp, int32_t* total_host) {
    cudaStream_t st = H.stream;
    const int64_t nblk = (n + 1023) / 1024;
    tmp.ensure(sizeof(int32_t) * (nblk + 2));
    if (n > 0) {
        k_scan_blocks<<<(int)nblk, 1024, 0, st>>>(in, n, out, tmp.as<int32_t>());
        k_scan_sums<<<1, 1024, 0, st>>>(tmp.as<int32_t>(), nblk, tmp.as<int32_t>() + nblk);
        k_scan_add<<<(int)nblk, 1024, 0, st>>>(out, n, tmp.as<int32_t>(), tmp.as<int32_t>() + nblk);
        GG_CUDA(cudaGetLastError());
        GG_CUDA(cudaMemcpyAsync(total_host, tmp.as<int32_t>() + nblk, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
    } else {
        *total_host = 0;
    }
    GG_CUDA(cudaStreamSynchronize(st));
}

// Locate + stable counting sort + gather.  Returns number of points outside the mesh.
int64_t locate_and_sort(Handle& H) {
    const int64_t np = H.np, nel = H.nel;
    cudaStream_t st = H.stream;
    H.offsets.ensure(sizeof(int32_t) * (nel + 1));
    H.fill.ensure(sizeof(int32_t) * (nel + 1));
    const int64_t nblk = (nel + 1023) / 1024;
    H.scan_tmp.ensure(sizeof(int32_t) * (nblk + 2));
    H.flag.ensure(sizeof(int32_t) * 4);
    GG_CUDA(cudaMemsetAsync(H.fill.p, 0, sizeof(int32_t) * (nel + 1), st));
    GG_CUDA(cudaMemsetAsync(H.flag.p, 0, sizeof(int32_t) * 4, st));
    // perm holds the points' places until k_segsort writes it
    k_locate<<<grid_for(np, 256), 256, 0, st>>>(H.mk, np, H.coords.as<double>(), H.cell.as<uint32_t>(),
                                                  H.fill.as<int32_t>(), H.flag.as<int32_t>(), H.perm.as<int32_t>());
    GG_CUDA(cudaGetLastError());
    k_scan_blocks<<<(int)nblk, 1024, 0, st>>>(H.fill.as<int32_t>(), nel, H.offsets.as<int32_t>(),
                                              H.scan_tmp.as<int32_t>());
    k_scan_sums<<<1, 1024, 0, st>>>(H.scan_tmp.as<int32_t>(), nblk, H.scan_tmp.as<int32_t>() + nblk);
    k_scan_add<<<(int)nblk, 1024, 0, st>>>(H.offsets.as<int32_t>(), nel, H.scan_tmp.as<int32_t>(),
                                           H.scan_tmp.as<int32_t>() + nblk);
    GG_CUDA(cudaGetLastError());
    // cell_s holds the unsorted permutation until k_segsort overwrites it
    launch_scatter(np, nel, H.cell.as<uint32_t>(), H.offsets.as<int32_t>(), H.perm.as<int32_t>(),
                   H.cell_s.as<int32_t>(), st);
    const int per = segsort_per(np, nel);
    k_segsort<false><<<segsort_grid(nel, per), kSegBlock, 0, st>>>(nel, per, H.offsets.as<int32_t>(),
                                                                   H.cell_s.as<int32_t>(), H.perm.as<int32_t>(),
                                                                   H.flag.as<int32_t>());
    GG_CUDA(cudaGetLastError());
    int32_t flags[2] = {0, 0};
    GG_CUDA(cudaMemcpyAsync(flags, H.flag.p, sizeof flags, cudaMemcpyDeviceToHost, st));
    GG_CUDA(cudaStreamSynchronize(st));
    const int32_t outside = flags[0];
    H.most_points = flags[1];
    const int64_t np_in = np - outside;
    k_gather_points<<<grid_for(np_in, 256), 256, 0, st>>>(
        H.mk, np_in, H.perm.as<int32_t>(), H.cell_s.as<int32_t>(), element_axes(H), H.coords.as<double>(),
        H.max_material > 0 ? H.mat_in.as<int32_t>() : nullptr, H.ps_given ? H.ps_in.as<double>() : nullptr,
        H.xi_s.as<double>(), H.mat_s.as<int32_t>(), H.ps_s.as<double>());
    GG_CUDA(cudaGetLastError());
    return outside;
}

}  // namespace gg
