// gg_cg64.cu -- the plain FP64 Jacobi CG (PETSc -ksp_type cg -pc_type jacobi, the inner
// solve of Stokes_SLE_UzawaSolver.cxx:554,620,725) as one persistent launch.
//
// What bounds it: on the meshes a plain FP64 solve is run on, one CG iteration is a
// microsecond of arithmetic, so the time is what separates its dependent steps.  As captured
// launches an iteration was 2^dim + 2 kernels (the apply needs one launch per element parity
// class to sum in a fixed order): 22-24 µs in 2D from 16² to 192², 54 µs on 16³ and 32³,
// whatever the arithmetic.  Here an iteration has two phases:
//   elements  p = z + βp formed at the gather, K_e p of every element stored per corner,
//             and the element energies pᵀK_e p;
//   nodes     α, each node adds its 2^dim element terms in class order (the sum the class
//             launches form), x, r, z, p, and the two dot products;
// so an iteration is two barriers.  2D meshes of up to about 64² run in the shared memory of
// one thread-block cluster (k_cg64_strip); others as a cooperative grid with the counter
// barrier of gg_grid.cuh (k_cg64).
// Every sum keeps the order of the launches it replaces (gg_solve.cu: 592 blocks of 256
// threads over the vectors, one block per 256-element tile of a class): the partial sums are
// formed per such block, by whichever CTA has it, and added in block index order by every
// CTA, so a solve gives the same bits on every run, for any number of CTAs.  Per iteration:
// 5.0 µs on 32², 5.1 on 64², 7.2 on 128², 13 on 16³, 19 on 32³, 38 on 48³ (60 as launches).
#include <math.h>

#include <algorithm>
#include <cstring>
#include <mutex>

#include "gg_cluster_addr.h"
#include "gg_grid.cuh"
#include "gg_internal.cuh"
#include "gg_kernels.cuh"
#include "gg_ops.cuh"

namespace gg {

namespace {

constexpr int kVecBlocks = 592;  // blocks of 256 threads the vector sums are split over
constexpr int kCluster = 16;
constexpr int kStripSmem = 222 * 1024;
constexpr int64_t kTermBytes = int64_t(32) << 20;  // element terms that stay in L2
// dofs of the solves under way at once from which they fill the GPU as launches
constexpr int64_t kSharedDofs2 = 1200000, kSharedDofs3 = 800000;

struct Cg64Args {
    MeshK mk;
    const double *mom, *b, *diag;
    const uint8_t* bc;
    double *x, *r, *z, *p;
    double* ye;     // element terms [class][corner·dim + component][element of the class]
    double* part_e; // [2^dim][tiles]: energy per element tile
    double* part_n; // [2][vec_blocks]: z·z and r·z per vector block
    KrylovScalars* s;
    GridBarrier* gb;
    double rtol;
    int maxit, tiles, vec_blocks, class_max;
};

// threads per CTA: two groups of 256 in 2D; one in 3D, whose FP64 element term needs more
// than 128 registers
template <int DIM>
constexpr int cg64_threads() { return DIM == 2 ? 512 : 256; }

__device__ __forceinline__ void group_bar(int g) {
    asm volatile("bar.sync %0, 256;" ::"r"(g + 1) : "memory");
}

// Sums of NV values over a group of 256 threads in block_sum's order; all threads get them.
template <int NV>
__device__ __forceinline__ void group_sum(double (&v)[NV], int g) {
    __shared__ double s_part[2][NV][8];
    __shared__ double s_tot[2][NV];
    const int lane = threadIdx.x & 31, wid = (threadIdx.x & 255) >> 5;
#pragma unroll
    for (int k = 0; k < NV; k++) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
        if (lane == 0) s_part[g][k][wid] = v[k];
    }
    group_bar(g);
    if (wid == 0) {
#pragma unroll
        for (int k = 0; k < NV; k++) {
            double t = lane < 8 ? s_part[g][k][lane] : 0.0;
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
            if (lane == 0) s_tot[g][k] = t;
        }
    }
    group_bar(g);
#pragma unroll
    for (int k = 0; k < NV; k++) v[k] = s_tot[g][k];
}

// element of thread t in tile `tile` of class `color` (apply_tiles_class)
struct ElemAt {
    int32_t e, n0, term;  // element, its corner 0 node, its index in the class's terms
    bool on;
};
template <int DIM>
__device__ __forceinline__ ElemAt elem_at(const Cg64Args& A, int unit, int t) {
    const MeshK& mk = A.mk;
    constexpr int TX = ApplyTile<DIM>::X, TY = ApplyTile<DIM>::Y, TZ = ApplyTile<DIM>::Z;
    const int color = unit / A.tiles, tile = unit - color * A.tiles;
    const int c0 = class_extent<DIM>(mk, 0, color), c1 = class_extent<DIM>(mk, 1, color);
    const int c2 = DIM == 3 ? class_extent<DIM>(mk, 2, color) : 1;
    const int ntx = (c0 + TX - 1) / TX, nty = (c1 + TY - 1) / TY, ntz = (c2 + TZ - 1) / TZ;
    ElemAt q{0, 0, 0, false};
    if (tile >= ntx * nty * ntz) return q;
    const int rr = tile / ntx;
    const int ci = (tile - rr * ntx) * TX + t % TX, cj = (rr % nty) * TY + (t / TX) % TY;
    const int ck = (rr / nty) * TZ + t / (TX * TY);
    if (ci >= c0 || cj >= c1 || ck >= c2) return q;
    const int i = 2 * ci + (color & 1), j = 2 * cj + ((color >> 1) & 1), k = DIM == 3 ? 2 * ck + ((color >> 2) & 1) : 0;
    q.e = i + mk.n[0] * (j + mk.n[1] * k);
    q.n0 = i + mk.nn[0] * (j + (DIM == 3 ? mk.nn[1] * k : 0));
    q.term = color * (1 << DIM) * DIM * A.class_max + ci + c0 * (cj + c1 * ck);
    q.on = true;
    return q;
}

// terms of vector entry i = c·nnode + n: one per class in class order, −1 where the node has
// no element of that class
template <int DIM>
struct NodeAt {
    int32_t term[1 << DIM];
    bool fixed;
};
template <int DIM>
__device__ __forceinline__ NodeAt<DIM> node_at(const Cg64Args& A, int64_t at) {
    const MeshK& mk = A.mk;
    const int c = (int)(at / mk.nnode);
    const int32_t n = (int32_t)(at - (int64_t)c * mk.nnode);
    const int i = n % mk.nn[0], rr = n / mk.nn[0];
    const int j = DIM == 3 ? rr % mk.nn[1] : rr, k = DIM == 3 ? rr / mk.nn[1] : 0;
    NodeAt<DIM> q;
    q.fixed = (A.bc[n] >> c) & 1;
#pragma unroll
    for (int color = 0; color < (1 << DIM); color++) {
        // the element of this class around the node has the node as its corner a
        const int ai = (i ^ color) & 1, aj = (j ^ (color >> 1)) & 1, ak = DIM == 3 ? (k ^ (color >> 2)) & 1 : 0;
        const int ei = i - ai, ej = j - aj, ek = k - ak;
        const bool in = ei >= 0 && ei < mk.n[0] && ej >= 0 && ej < mk.n[1] && (DIM == 2 || (ek >= 0 && ek < mk.n[2]));
        const int c0 = class_extent<DIM>(mk, 0, color), c1 = class_extent<DIM>(mk, 1, color);
        const int a = ai | (aj << 1) | (ak << 2);
        q.term[color] = in ? ((color * (1 << DIM) + a) * DIM + c) * A.class_max + (ei >> 1) +
                                 c0 * ((ej >> 1) + c1 * (DIM == 3 ? ek >> 1 : 0))
                           : -1;
    }
    return q;
}

template <int DIM>
__global__ void __launch_bounds__(cg64_threads<DIM>(), 1) k_cg64(const __grid_constant__ Cg64Args A) {
    constexpr int NS = 1 << DIM, NM = n_moments<DIM>();
    const MeshK& mk = A.mk;
    const int64_t nnode = mk.nnode, n = (int64_t)DIM * nnode;
    constexpr int64_t kStride = (int64_t)kVecBlocks * 256;
    const int g = threadIdx.x >> 8, t = threadIdx.x & 255;
    // the first gridDim.x tiles and vector blocks go to different SMs
    const int slot = g * gridDim.x + blockIdx.x, slots = gridDim.x * (cg64_threads<DIM>() / 256);
    const int units = NS * A.tiles;
    unsigned int epoch = 0;
    int32_t rowoff[NS];
#pragma unroll
    for (int a = 0; a < NS; a++)
        rowoff[a] = (a & 1) + ((a >> 1) & 1) * mk.nn[0] + (DIM == 3 ? ((a >> 2) & 1) * mk.nn[0] * mk.nn[1] : 0);

    // x = 0, r = b, z = D⁻¹r (k_cg_init); p = 0 with β = 0 makes the first direction z
    for (int u = slot; u < units; u += slots)
        if (t == 0) A.part_e[u] = 0.0;
    for (int vb = slot; vb < A.vec_blocks; vb += slots) {
        double acc[2] = {0.0, 0.0};
        for (int64_t i = (int64_t)vb * 256 + t; i < n; i += kStride) {
            const int c = (int)(i / nnode);
            const bool fixed = (A.bc[i - (int64_t)c * nnode] >> c) & 1;
            const double rv = fixed ? 0.0 : A.b[i];
            const double zv = fixed ? 0.0 : rv / A.diag[i];
            A.x[i] = 0.0;
            A.r[i] = rv;
            A.z[i] = zv;
            A.p[i] = 0.0;
            acc[0] += zv * zv;
            acc[1] += rv * zv;
        }
        group_sum<2>(acc, g);
        if (t == 0) {
            A.part_n[vb] = acc[0];
            A.part_n[A.vec_blocks + vb] = acc[1];
        }
    }
    if (!grid_barrier(A.gb, &epoch)) return;
    auto vec_sums = [&](double (&v)[2]) {
        v[0] = v[1] = 0.0;
        for (int b = t; b < A.vec_blocks; b += 256) {
            v[0] += __ldcg(A.part_n + b);
            v[1] += __ldcg(A.part_n + A.vec_blocks + b);
        }
        group_sum<2>(v, g);
    };
    // a thread's first element and first vector entry do not change over the iterations
    const ElemAt first_e = slot < units ? elem_at<DIM>(A, slot, t) : ElemAt{0, 0, 0, false};
    const int64_t first_i = (int64_t)slot * 256 + t;
    const bool have_n = slot < A.vec_blocks && first_i < n;
    const NodeAt<DIM> first_n = node_at<DIM>(A, have_n ? first_i : 0);
    const double first_d = have_n ? A.diag[first_i] : 1.0;

    double beta = 0.0, rz = 0.0, rnorm = 0.0, rnorm0 = 0.0, ttol = 0.0, pAp = 0.0;
    int it = 0, failed = 0;
    bool started = false;
    for (;;) {
        // ---- elements.  The loads of the first element do not depend on β
        double zz[DIM][NS], pp[DIM][NS], M[NM];
        auto load_elem = [&](const ElemAt& q) {
#pragma unroll
            for (int c = 0; c < DIM; c++)
#pragma unroll
                for (int a = 0; a < NS; a++) {
                    zz[c][a] = __ldcg(A.z + c * nnode + q.n0 + rowoff[a]);
                    pp[c][a] = __ldcg(A.p + c * nnode + q.n0 + rowoff[a]);
                }
#pragma unroll
            for (int k = 0; k < NM; k++) M[k] = __ldg(A.mom + (int64_t)k * mk.nel + q.e);
        };
        if (first_e.on) load_elem(first_e);
        double sums[2];
        vec_sums(sums);
        if (started) beta = sums[1] / rz;
        rz = sums[1];
        for (int u = slot; u < units; u += slots) {
            ElemAt q = first_e;
            if (u != slot) {
                q = elem_at<DIM>(A, u, t);
                if (q.on) load_elem(q);
            }
            double en[1] = {0.0};
            if (q.on) {
                double m[DIM][NS];
#pragma unroll
                for (int c = 0; c < DIM; c++)
#pragma unroll
                    for (int a = 0; a < NS; a++) m[c][a] = zz[c][a] + beta * pp[c][a];
                en[0] = element_compute<DIM, double, true>(mk, m, M, -1, [&](int c, int row, double v0, double v1) {
                    __stcg(A.ye + q.term + (int64_t)(2 * row * DIM + c) * A.class_max, v0);
                    __stcg(A.ye + q.term + (int64_t)((2 * row + 1) * DIM + c) * A.class_max, v1);
                });
            }
            group_sum<1>(en, g);
            if (t == 0) A.part_e[u] = en[0];
        }
        // the stopping test, behind the element terms so that the square root is off the
        // iteration's chain (terms of an iteration that does not happen are never read)
        rnorm = sqrt(sums[0]);
        if (!started) {
            started = true;
            rnorm0 = rnorm;
            const double tt = A.rtol * rnorm0;
            ttol = tt < 1e-50 ? 1e-50 : tt;
            if (rnorm0 <= ttol) break;
        } else {
            it++;
            if (!(rnorm == rnorm) || isinf(rnorm)) {
                failed = 2;
                break;
            }
            if (rnorm <= ttol) break;
            if (it >= A.maxit) {
                failed = 1;
                break;
            }
        }
        if (!grid_barrier(A.gb, &epoch)) return;
        // ---- nodes.  The loads of the first entry do not depend on α
        double ye[NS], rv = 0.0, zv = 0.0, pv = 0.0, xv = 0.0;
        auto load_node = [&](const NodeAt<DIM>& q, int64_t i) {
#pragma unroll
            for (int k = 0; k < NS; k++) ye[k] = q.term[k] >= 0 ? __ldcg(A.ye + q.term[k]) : 0.0;
            rv = A.r[i];
            xv = A.x[i];
            zv = __ldcg(A.z + i);
            pv = __ldcg(A.p + i);
        };
        if (have_n) load_node(first_n, first_i);
        double e[1] = {0.0};
        for (int b = t; b < units; b += 256) e[0] += __ldcg(A.part_e + b);
        group_sum<1>(e, g);
        pAp = e[0];
        const double alpha = rz / pAp;
        if (!(pAp > 0.0) || isinf(pAp)) {
            failed = 3;
            break;
        }
        for (int vb = slot; vb < A.vec_blocks; vb += slots) {
            double acc[2] = {0.0, 0.0};
            for (int64_t i = (int64_t)vb * 256 + t; i < n; i += kStride) {
                NodeAt<DIM> q = first_n;
                double d = first_d;
                if (i != first_i) {
                    q = node_at<DIM>(A, i);
                    d = A.diag[i];
                    load_node(q, i);
                }
                double ap = 0.0;
#pragma unroll
                for (int k = 0; k < NS; k++) ap += ye[k];
                const double pn = zv + beta * pv;
                A.x[i] = xv + alpha * pn;
                const double rn = q.fixed ? 0.0 : rv - alpha * ap;
                const double zn = q.fixed ? 0.0 : rn / d;
                A.r[i] = rn;
                __stcg(A.z + i, zn);
                __stcg(A.p + i, pn);
                acc[0] += zn * zn;
                acc[1] += rn * zn;
            }
            group_sum<2>(acc, g);
            if (t == 0) {
                A.part_n[vb] = acc[0];
                A.part_n[A.vec_blocks + vb] = acc[1];
            }
        }
        if (!grid_barrier(A.gb, &epoch)) return;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        A.s->rnorm0 = rnorm0;
        A.s->rnorm = rnorm;
        A.s->pAp = pAp;
        A.s->iterations = it;
        A.s->failed = failed;
        A.s->done = 1;
    }
}

// ---- 2D meshes whose strips fit the shared memory of one cluster ------------------------
// The same two phases with everything in shared memory: CTA s of the cluster owns the element
// rows R_s … R_{s+1} − 1 (even R_s, so every parity class keeps whole rows) and, of the vector
// entries, an equal share of the 32-entry chunks at about the same nodes.  A phase writes what the next
// one reads straight into the reader's shared memory: an element its corner terms to the CTA
// that sums that entry, an entry its z and p to the one or two strips whose elements use its
// node -- nearly always the CTA itself, where a plain store does (a store through the cluster
// window moves some 16 bytes per cycle and CTA, and 18 warps that each stored their sums to
// 16 CTAs took 2000 cycles).  The partial sums go to every CTA in one contiguous piece per
// destination.  An iteration is then two cluster barriers of 450 cycles, the two divisions,
// the sums, and no load from L2: 5.0 µs on 20² to 48², 5.1 on 64², where the grid form takes
// 7.0-7.6 and the captured launches 22-24.  What is left is the instruction latency of the
// one warp per scheduler that has work (the element term alone is 1400 cycles).
// The sums: a warp of k_cg64's 256-thread blocks is one class row segment of 32 elements, or
// one chunk of 32 vector entries, so the partial sums exchanged are those of the warps, and
// they are added up in block_sum's order.
constexpr int kStripThreads = 576;  // 18 warps of ≤ 112 registers: a 64² strip has 17-18 chunks

struct Cg64Strip {
    int cluster;
    int row[kCluster + 1];              // first element row of every strip
    int max_tasks, max_chunks, max_nl;  // array extents, the same in every CTA
    int units, vec_blocks;              // element tiles, vector blocks of 256
    // byte offsets in shared memory
    int zl, pl, terms, x, r, d, z, p, mom, taddr, zaddr, ex, nx, ei, ni, bytes;
};

__device__ __forceinline__ unsigned shared_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
// address of p in the cluster's CTA `rank`, marked as remote; in this CTA (`me`) the plain
// shared address
__device__ __forceinline__ unsigned cluster_addr(const void* p, int rank, int me) {
    const unsigned a = shared_addr(p);
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return rank == me ? a : mark_remote(r);
}
// the mark comes off in the address offset
__device__ __forceinline__ void cluster_store(unsigned a, double v) {
    static_assert(kRemoteBit == 1u, "the offset of the remote store");
    asm volatile(
        "{\n\t.reg .pred r;\n\t"
        "setp.ne.u32 r, %1, 0;\n\t"
        "@r st.shared::cluster.f64 [%0+-1], %2;\n\t@!r st.shared::cta.f64 [%0], %2;\n\t}" ::"r"(a),
        "r"(a & kRemoteBit), "d"(v)
        : "memory");
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// CTA s owns the chunks of component c that begin at nodes s·nnode/cluster … (equal shares, so
// the last strip's extra node row makes no CTA wait); the first of them
__device__ __forceinline__ int chunk_lo(const MeshK& mk, const Cg64Strip& S, int s, int c) {
    return (int)((c * mk.nnode + s * mk.nnode / S.cluster + 31) >> 5);
}
__device__ __forceinline__ int chunk_owner(const MeshK& mk, const Cg64Strip& S, int node) {
    int s = 0;
    while (s + 1 < S.cluster && node >= (int)((s + 1) * mk.nnode / S.cluster)) s++;
    return s;
}
// strip of a node row
__device__ __forceinline__ int strip_of(const Cg64Strip& S, int node_row) {
    int s = 0;
    while (s + 1 < S.cluster && node_row >= S.row[s + 1]) s++;
    return s;
}

// Sum over up to 256 blocks of NV values, each block the block_sum of its 8 warps' partial
// sums v[idx[8b + w]], as the last block of a 256-thread launch forms it: a CTA warp per launch warp, then
// every thread adds up the warps.  stage: [8·NV] doubles, zero past the launch's warps; the
// CTA meets once.
template <int NV>
__device__ __forceinline__ void cta_total(const double* v, const uint16_t* idx, int blocks, double* stage,
                                          double (&tot)[NV]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (32 * warp < blocks) {
        const uint4 at = *reinterpret_cast<const uint4*>(idx + 8 * threadIdx.x);  // a zero past the blocks
        const uint32_t pair[4] = {at.x, at.y, at.z, at.w};
        double p[8][NV], s[NV];
#pragma unroll
        for (int w = 0; w < 8; w++) {
            const int q = (pair[w >> 1] >> (16 * (w & 1))) & 0xffff;
#pragma unroll
            for (int k = 0; k < NV; k++) p[w][k] = v[q * NV + k];
        }
#pragma unroll
        for (int k = 0; k < NV; k++)
            s[k] = ((p[0][k] + p[4][k]) + (p[2][k] + p[6][k])) + ((p[1][k] + p[5][k]) + (p[3][k] + p[7][k]));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int k = 0; k < NV; k++) s[k] += __shfl_xor_sync(0xffffffffu, s[k], o);
        if (lane == 0)
#pragma unroll
            for (int k = 0; k < NV; k++) stage[8 * k + warp] = s[k];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NV; k++) {
        const double* t = stage + 8 * k;
        tot[k] = ((t[0] + t[4]) + (t[2] + t[6])) + ((t[1] + t[5]) + (t[3] + t[7]));
    }
}

__global__ void __launch_bounds__(kStripThreads, 1)
k_cg64_strip(const __grid_constant__ Cg64Args A, const __grid_constant__ Cg64Strip S) {
    extern __shared__ __align__(16) unsigned char sm[];
    __shared__ double stage_n[16], stage_e[8];
    __shared__ int s_stop;  // 0 go on, 1 converged, 2 iteration limit, 3 not finite
    constexpr int NS = 4, NM = 6, kWarps = kStripThreads / 32;
    static_assert(kWarps >= kCluster, "a warp per destination");
    const MeshK& mk = A.mk;
    const int nnode = (int)mk.nnode, n = 2 * nnode, nn0 = mk.nn[0];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int me = blockIdx.x;  // one cluster: the CTA's rank in it
    const int r0 = S.row[me], r1 = S.row[me + 1];
    // [2][max_nl]: node rows r0 … r1, the even nodes of a row before the odd ones, so that the
    // elements of a class read neighbouring words
    double* zl = reinterpret_cast<double*>(sm + S.zl);
    const int half = (nn0 + 1) / 2;
    double* pl = reinterpret_cast<double*>(sm + S.pl);
    double* terms = reinterpret_cast<double*>(sm + S.terms);  // [4 classes][32·max_chunks]
    double* xs = reinterpret_cast<double*>(sm + S.x);         // the CTA's entries
    double* rs = reinterpret_cast<double*>(sm + S.r);
    double* ds = reinterpret_cast<double*>(sm + S.d);
    double* zs = reinterpret_cast<double*>(sm + S.z);
    double* ps = reinterpret_cast<double*>(sm + S.p);
    double* mom = reinterpret_cast<double*>(sm + S.mom);          // [6][32·max_tasks]
    unsigned* taddr = reinterpret_cast<unsigned*>(sm + S.taddr);  // [8][32·max_tasks]
    unsigned* zaddr = reinterpret_cast<unsigned*>(sm + S.zaddr);  // [2][32·max_chunks], then: entry fixed or missing
    // partial sums of every CTA: element tasks [cluster][max_tasks], chunks
    // [cluster][max_chunks][2], a zero behind each; where those of a block's 8 warps are
    double* ex = reinterpret_cast<double*>(sm + S.ex);
    double* nx = reinterpret_cast<double*>(sm + S.nx);
    uint16_t* ei = reinterpret_cast<uint16_t*>(sm + S.ei);  // [units][8]
    uint16_t* ni = reinterpret_cast<uint16_t*>(sm + S.ni);  // [vec_blocks][8]
    const int te_n = 32 * S.max_tasks, ts_n = 32 * S.max_chunks;
    // this CTA's chunks: component 0, then component 1
    const int q0 = chunk_lo(mk, S, me, 0), c0n = chunk_lo(mk, S, me + 1, 0) - q0;
    const int q1 = chunk_lo(mk, S, me, 1), chunks = c0n + chunk_lo(mk, S, me + 1, 1) - q1;
    // its element tasks: (class row pair of the strip, class, segment of 32)
    const int ntx0 = ((mk.n[0] + 1) / 2 + 31) / 32, tasks = (r1 - r0 + 1) / 2 * 4 * ntx0;
    const unsigned off_pl = (unsigned)(S.pl - S.zl);

    // ---- tables
    for (int i = threadIdx.x; i < 4 * ts_n; i += kStripThreads) terms[i] = 0.0;
    for (int i = threadIdx.x; i < 8 * ((S.units + 31) & ~31); i += kStripThreads) ei[i] = (uint16_t)(S.cluster * S.max_tasks);
    for (int i = threadIdx.x; i < 8 * ((S.vec_blocks + 31) & ~31); i += kStripThreads) ni[i] = (uint16_t)(S.cluster * S.max_chunks);
    if (threadIdx.x < 16) stage_n[threadIdx.x] = 0.0;
    if (threadIdx.x < 8) stage_e[threadIdx.x] = 0.0;
    if (threadIdx.x == 0) {
        ex[S.cluster * S.max_tasks] = 0.0;
        nx[2 * S.cluster * S.max_chunks] = nx[2 * S.cluster * S.max_chunks + 1] = 0.0;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < S.cluster * S.max_tasks; i += kStripThreads) {
        // tile of the class row: rows in eights, segments of the class's own width
        const int s = i / S.max_tasks, task = i - s * S.max_tasks;
        const int seg = task % ntx0, color = (task / ntx0) & 3, cj = S.row[s] / 2 + task / (4 * ntx0);
        const int ntx = (class_extent<2>(mk, 0, color) + 31) / 32;
        if (task < (S.row[s + 1] - S.row[s] + 1) / 2 * 4 * ntx0 && seg < ntx)
            ei[8 * (color * A.tiles + (cj >> 3) * ntx + seg) + (cj & 7)] = (uint16_t)i;
    }
    for (int i = threadIdx.x; i < S.cluster * S.max_chunks; i += kStripThreads) {
        const int s = i / S.max_chunks, slot = i - s * S.max_chunks;
        const int a0 = chunk_lo(mk, S, s, 0), n0 = chunk_lo(mk, S, s + 1, 0) - a0;
        const int a1 = chunk_lo(mk, S, s, 1), n1 = chunk_lo(mk, S, s + 1, 1) - a1;
        if (slot < n0 + n1) ni[slot < n0 ? a0 + slot : a1 + slot - n0] = (uint16_t)i;
    }
    for (int te = threadIdx.x; te < te_n; te += kStripThreads) {
        const int task = te >> 5, seg = task % ntx0, color = (task / ntx0) & 3, cj = r0 / 2 + task / (4 * ntx0);
        const int i = 2 * (32 * seg + (te & 31)) + (color & 1), j = 2 * cj + (color >> 1);
        const bool on = task < tasks && i < mk.n[0] && j < r1;
        for (int a = 0; a < NS; a++) {
            const int node = i + (a & 1) + nn0 * (j + (a >> 1));
            for (int c = 0; c < 2; c++) {
                unsigned t = kNoAddr;
                if (on) {
                    const int at = c * nnode + node, q = at >> 5, first = q << 5;
                    const int fc = first >= nnode ? 1 : 0, s = chunk_owner(mk, S, first - fc * nnode);
                    const int lo = chunk_lo(mk, S, s, 0);
                    const int slot = fc == 0 ? q - lo : chunk_lo(mk, S, s + 1, 0) - lo + q - chunk_lo(mk, S, s, 1);
                    t = cluster_addr(terms + color * ts_n + slot * 32 + (at & 31), s, me);
                }
                taddr[(a * 2 + c) * te_n + te] = t;
            }
        }
        if (on)
            for (int k = 0; k < NM; k++) mom[k * te_n + te] = A.mom[(int64_t)k * mk.nel + i + mk.n[0] * j];
    }
    for (int ts = threadIdx.x; ts < ts_n; ts += kStripThreads) {
        const int slot = ts >> 5, at = 32 * (slot < c0n ? q0 + slot : q1 + slot - c0n) + (ts & 31);
        unsigned t0 = kNoAddr, t1 = kNoAddr;
        if (slot < chunks && at < n) {
            const int c = at >= nnode, node = at - c * nnode, row = node / nn0, s = strip_of(S, row);
            const int col = node % nn0, at_l = c * S.max_nl + (col & 1) * half + (col >> 1);
            t0 = cluster_addr(zl + at_l + (row - S.row[s]) * nn0, s, me);
            if (s > 0 && row == S.row[s])
                t1 = cluster_addr(zl + at_l + (row - S.row[s - 1]) * nn0, s - 1, me);
        }
        zaddr[ts] = t0;
        zaddr[ts_n + ts] = t1;
    }
    cluster_barrier();  // every CTA's arrays exist and are zeroed
    // z and p of entry ts to the strips that gather it
    auto publish = [&](int ts, double zv, double pv) {
        const unsigned t0 = zaddr[ts], t1 = zaddr[ts_n + ts];
        if (t0 != kNoAddr) {
            cluster_store(t0, zv);
            cluster_store(t0 + off_pl, pv);
        }
        if (t1 != kNoAddr) {
            cluster_store(t1, zv);
            cluster_store(t1 + off_pl, pv);
        }
    };
    // this CTA's `count` doubles at own[0 …] to the same place of every other CTA, a warp each
    auto share = [&](const double* own, int count) {
        __syncthreads();
        if (warp < S.cluster && warp != me) {
            const unsigned t = cluster_addr(own, warp, me);
            for (int k = lane; k < count; k += 32) cluster_store(t + 8u * (unsigned)k, own[k]);
        }
    };
    double* own_n = nx + 2 * me * S.max_chunks;
    double* own_e = ex + me * S.max_tasks;
    // the two sums of the warp's chunk
    auto chunk_sums = [&](int slot, double a, double b) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            a += __shfl_xor_sync(0xffffffffu, a, o);
            b += __shfl_xor_sync(0xffffffffu, b, o);
        }
        if (lane == 0) {
            own_n[2 * slot] = a;
            own_n[2 * slot + 1] = b;
        }
    };
    for (int slot = warp; slot < chunks; slot += kWarps) {
        const int ts = slot * 32 + lane, at = 32 * (slot < c0n ? q0 + slot : q1 + slot - c0n) + lane;
        double zz = 0.0, rz = 0.0, rv = 0.0, zv = 0.0, dv = 1.0;
        bool fixed = true;
        if (at < n) {
            const int c = at >= nnode;
            fixed = (A.bc[at - c * nnode] >> c) & 1;
            if (!fixed) {
                dv = A.diag[at];
                rv = A.b[at];
                zv = rv / dv;
            }
            zz = zv * zv;
            rz = rv * zv;
        }
        xs[ts] = 0.0;
        rs[ts] = rv;
        ds[ts] = dv;
        zs[ts] = zv;
        ps[ts] = 0.0;
        zaddr[2 * ts_n + ts] = fixed;
        publish(ts, zv, 0.0);
        chunk_sums(slot, zz, rz);
    }
    share(own_n, 2 * chunks);
    cluster_barrier();

    // local node of a task's element, and what does not change over the iterations
    auto elem_nz = [&](int task) {
        const int seg = task % ntx0, color = (task / ntx0) & 3, lp = task / (4 * ntx0);
        const int px = color & 1;  // its corner 0; the next node of the row: (see load_elem)
        return 32 * seg + lane + px * half + nn0 * (2 * lp + (color >> 1));
    };
    const int first_nz = elem_nz(warp);
    const bool first_on = warp < tasks && taddr[warp * 32 + lane] != kNoAddr;

    double beta = 0.0, rz = 0.0, rnorm = 0.0, rnorm0 = 0.0, ttol = 0.0, pAp = 0.0;
    int it = 0, failed = 0;
    bool started = false;
    for (;;) {
        // ---- elements (the first task's loads do not wait for β)
        double zz[2][NS], pp[2][NS], M[NM];
        auto load_elem = [&](int nz, int task, int te) {
            // the odd neighbour of an even node, the even neighbour of an odd one
            const int dx = ((task / ntx0) & 1) ? 1 - half : half;
#pragma unroll
            for (int c = 0; c < 2; c++)
#pragma unroll
                for (int a = 0; a < NS; a++) {
                    const int at = c * S.max_nl + nz + (a & 1) * dx + nn0 * (a >> 1);
                    zz[c][a] = zl[at];
                    pp[c][a] = pl[at];
                }
#pragma unroll
            for (int k = 0; k < NM; k++) M[k] = mom[k * te_n + te];
        };
        if (first_on) load_elem(first_nz, warp, warp * 32 + lane);
        double sums[2];
        cta_total<2>(nx, ni, S.vec_blocks, stage_n, sums);
        if (started) beta = sums[1] / rz;
        rz = sums[1];
        for (int task = warp; task < tasks; task += kWarps) {
            const int te = task * 32 + lane;
            const bool on = task == warp ? first_on : taddr[te] != kNoAddr;
            if (on && task != warp) load_elem(elem_nz(task), task, te);
            double en = 0.0;
            if (on) {
                double m[2][NS];
#pragma unroll
                for (int c = 0; c < 2; c++)
#pragma unroll
                    for (int a = 0; a < NS; a++) m[c][a] = zz[c][a] + beta * pp[c][a];
                en = element_compute<2, double, true>(mk, m, M, -1, [&](int c, int row, double v0, double v1) {
                    cluster_store(taddr[(4 * row + c) * te_n + te], v0);
                    cluster_store(taddr[(4 * row + 2 + c) * te_n + te], v1);
                });
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) en += __shfl_xor_sync(0xffffffffu, en, o);
            if (lane == 0) own_e[task] = en;
        }
        if (warp == kWarps - 1) {
            // the stopping test, by the warp that has the fewest tasks
            rnorm = sqrt(sums[0]);
            if (!started) {
                rnorm0 = rnorm;
                const double tt = A.rtol * rnorm0;
                ttol = tt < 1e-50 ? 1e-50 : tt;
            }
            const int done = it + (started ? 1 : 0);
            if (lane == 0)
                s_stop = started && (!(rnorm == rnorm) || isinf(rnorm)) ? 3
                         : rnorm <= ttol                                ? 1
                         : started && done >= A.maxit                   ? 2
                                                                        : 0;
        }
        share(own_e, tasks);
        if (started) it++;
        started = true;
        if (s_stop) {
            failed = s_stop - 1;
            break;
        }
        cluster_barrier();
        // ---- nodes (the first chunk's loads do not wait for α)
        double ye[NS], rv, xv, zv, pv;
        auto load_node = [&](int ts) {
#pragma unroll
            for (int k = 0; k < NS; k++) ye[k] = terms[k * ts_n + ts];
            rv = rs[ts];
            xv = xs[ts];
            zv = zs[ts];
            pv = ps[ts];
        };
        if (warp < chunks) load_node(warp * 32 + lane);
        double e[1];
        cta_total<1>(ex, ei, S.units, stage_e, e);
        pAp = e[0];
        const double alpha = rz / pAp;
        if (!(pAp > 0.0) || isinf(pAp)) {
            failed = 3;
            break;
        }
        for (int slot = warp; slot < chunks; slot += kWarps) {
            const int ts = slot * 32 + lane;
            if (slot != warp) load_node(ts);
            const bool fixed = zaddr[2 * ts_n + ts] != 0u;
            double ap = 0.0;
#pragma unroll
            for (int k = 0; k < NS; k++) ap += ye[k];
            const double pnew = zv + beta * pv;
            xs[ts] = xv + alpha * pnew;
            const double rn = fixed ? 0.0 : rv - alpha * ap;
            const double zn = fixed ? 0.0 : rn / ds[ts];
            rs[ts] = rn;
            zs[ts] = zn;
            ps[ts] = pnew;
            publish(ts, zn, pnew);
            chunk_sums(slot, zn * zn, rn * zn);
        }
        share(own_n, 2 * chunks);
        cluster_barrier();
    }
    cluster_barrier();  // no CTA leaves while another may still write into it
    for (int slot = warp; slot < chunks; slot += kWarps) {
        const int at = 32 * (slot < c0n ? q0 + slot : q1 + slot - c0n) + lane;
        if (at < n) A.x[at] = xs[slot * 32 + lane];
    }
    if (me == 0 && threadIdx.x == kStripThreads - 32) {
        A.s->rnorm0 = rnorm0;
        A.s->rnorm = rnorm;
        A.s->pAp = pAp;
        A.s->iterations = it;
        A.s->failed = failed;
        A.s->done = 1;
    }
}

// Launch of the strip kernel; false where the mesh or the device does not allow it.
bool run_strip(Handle& H, const Cg64Args& A) {
    const MeshK& mk = H.mk;
    Cg64Strip S;
    std::memset(&S, 0, sizeof S);
    const int ny = mk.n[1], nn0 = mk.nn[0], pairs = (ny + 1) / 2;
    S.cluster = 1;
    while (2 * S.cluster <= kCluster && 2 * S.cluster <= pairs) S.cluster *= 2;
    for (int s = 0; s < S.cluster; s++) S.row[s] = 2 * (int)((int64_t)s * pairs / S.cluster);
    S.row[S.cluster] = ny;
    const int64_t nnode = mk.nnode;
    auto lo = [&](int s, int c) {
        return (c * nnode + s * nnode / S.cluster + 31) / 32;
    };
    int64_t tasks = 0, chunks = 0, nl = 0;
    for (int s = 0; s < S.cluster; s++) {
        const int rows = S.row[s + 1] - S.row[s];
        tasks = std::max<int64_t>(tasks, (int64_t)((rows + 1) / 2) * 4 * (((mk.n[0] + 1) / 2 + 31) / 32));
        chunks = std::max(chunks, lo(s + 1, 0) - lo(s, 0) + lo(s + 1, 1) - lo(s, 1));
        nl = std::max<int64_t>(nl, (int64_t)(rows + 1) * nn0);
    }
    int64_t at = 0;
    auto take = [&](int64_t bytes) {
        const int64_t r = at;
        at += (bytes + 15) / 16 * 16;
        return (int)std::min<int64_t>(r, 1 << 30);
    };
    const int64_t d = sizeof(double), te = 32 * tasks, ts = 32 * chunks;
    S.units = 4 * A.tiles;
    S.vec_blocks = A.vec_blocks;
    S.zl = take(2 * nl * d);
    S.pl = take(2 * nl * d);
    S.terms = take(4 * ts * d);
    S.x = take(ts * d);
    S.r = take(ts * d);
    S.d = take(ts * d);
    S.z = take(ts * d);
    S.p = take(ts * d);
    S.mom = take(6 * te * d);
    S.taddr = take(8 * te * 4);
    S.zaddr = take(3 * ts * 4);
    S.ex = take((S.cluster * tasks + 1) * d);
    S.nx = take((S.cluster * chunks + 1) * 2 * d);
    S.ei = take(8 * (int64_t)((S.units + 31) & ~31) * 2);  // whole warps read them
    S.ni = take(8 * (int64_t)((S.vec_blocks + 31) & ~31) * 2);
    // a second round of chunks costs what the cluster gains: 72² (21 chunks per CTA) 7.4 µs per
    // iteration against 7.6 as a grid, 96² 8.5 against 7.4
    if (chunks > kStripThreads / 32) return false;
    if (at > kStripSmem || S.cluster * std::max(tasks, chunks) >= 65535 || S.units > 256 || S.vec_blocks > 256) return false;
    S.bytes = (int)at;
    S.max_tasks = (int)tasks;
    S.max_chunks = (int)chunks;
    S.max_nl = (int)nl;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(S.cluster);
    cfg.blockDim = dim3(kStripThreads);
    cfg.dynamicSmemBytes = S.bytes;
    cfg.stream = H.stream;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = S.cluster;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int fits = 0;
    if (cudaFuncSetAttribute(k_cg64_strip, cudaFuncAttributeMaxDynamicSharedMemorySize, kStripSmem) != cudaSuccess ||
        cudaFuncSetAttribute(k_cg64_strip, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&fits, (const void*)k_cg64_strip, &cfg) != cudaSuccess || fits < 1) {
        cudaGetLastError();
        return false;
    }
    GG_CUDA(cudaLaunchKernelEx(&cfg, k_cg64_strip, A, S));
    return true;
}

template <int DIM>
int run(Handle& H, Cg64Args& A, int solves) {
    if (DIM == 2 && H.cg64_form != 2 && run_strip(H, A)) return 0;
    constexpr int T = cg64_threads<DIM>(), per = T / 256;
    const int work = std::max(A.tiles << DIM, A.vec_blocks);
    const void* fn = (const void*)k_cg64<DIM>;
    int per_sm = 0;
    GG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, T, 0));
    if (per_sm < 1) return 1;
    // its share of the SMs beside other solves, whose grids then run at the same time
    const int grid = std::min((work + per - 1) / per, std::max(1, per_sm * num_sms() / solves));
    GG_CUDA(cudaMemsetAsync(A.gb, 0, sizeof(GridBarrier), H.stream));
    void* args[] = {(void*)&A};
    GG_CUDA(cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(T), args, 0, H.stream));
    return 0;
}

struct InFlight {
    std::mutex mu;
    int solves = 0;
    int64_t dofs = 0;
};
InFlight& in_flight(int dev) {
    static InFlight f[64];
    return f[dev >= 0 && dev < 64 ? dev : 0];
}

}  // namespace

Fp64Flight::Fp64Flight(const Handle& H) : dev(H.device), mine(H.ndof) {
    InFlight& f = in_flight(dev);
    std::lock_guard<std::mutex> lk(f.mu);
    solves = ++f.solves;
    dofs = f.dofs += mine;
}
Fp64Flight::~Fp64Flight() {
    InFlight& f = in_flight(dev);
    std::lock_guard<std::mutex> lk(f.mu);
    f.solves--;
    f.dofs -= mine;
}

// x = K⁻¹ b to ‖D⁻¹r‖ ≤ max(rtol‖D⁻¹b‖, 1e-50) in FP64.  Returns 1 when the mesh is outside
// this kernel's limits (element terms beyond kTermBytes, or a class of more tiles than the
// class launches have blocks): the caller then runs the captured launches.
//
// Solves from several threads (gg_solve_batch, or a caller's own) share the device.  A
// cooperative grid on every SM would make them take turns, so each takes its share; and where
// together they are large enough to fill the GPU, the launches, which interleave freely, do more
// per second (ms of a batch, launches / turns / shares: 16 of 128² 506 / 466 / 330, of 192² 904 / 1364 /
// 809, of 24³ 318 / 415 / 292, of 32³ 676 / 886 / 817, 8 of 48³ 1189 / 1460 / 1612, of 400² 2744 /
// 3094 / 2936; 4 at a time of 32³ 843 / 892 / 728, of 256² 2149 / 2552 / 1636).  The bits are the
// same in every form.
int run_cg64(Handle& H, const Fp64Flight& flight, const double* b, double* x, double rtol, int maxit, int* iters) {
    const int dim = H.dim, nc = 1 << dim;
    if (H.cg64_form == 1 || (H.cg64_form == 0 && flight.solves > 1 && flight.dofs > (dim == 2 ? kSharedDofs2 : kSharedDofs3)))
        return 1;
    int64_t class_max = 0;
    int tiles = 1;
    for (int c = 0; c < nc; c++) {
        int64_t m = 1, tl = 0;
        for (int d = 0; d < dim; d++) m *= (H.mk.n[d] - ((c >> d) & 1) + 1) >> 1;
        class_max = std::max(class_max, m);
        tl = dim == 3 ? class_tiles<3>(H.mk, c, ApplyTile<3>::X, ApplyTile<3>::Y, ApplyTile<3>::Z)
                      : class_tiles<2>(H.mk, c, ApplyTile<2>::X, ApplyTile<2>::Y, ApplyTile<2>::Z);
        if (tl > class_grid(H.mk, c)) return 1;
        tiles = std::max(tiles, class_grid(H.mk, c));
    }
    const int64_t terms = (int64_t)nc * nc * dim * class_max;
    if ((int64_t)sizeof(double) * terms > kTermBytes) return 1;
    Cg64Args A;
    std::memset(&A, 0, sizeof A);
    A.mk = H.mk;
    A.mom = H.mom64.as<double>();
    A.b = b;
    A.diag = H.kdiag64.as<double>();
    A.bc = H.bcmask.as<uint8_t>();
    A.x = x;
    A.r = H.cg_r.as<double>();
    A.z = H.cg_z.as<double>();
    A.p = H.cg_p.as<double>();
    A.rtol = rtol;
    A.maxit = maxit;
    A.tiles = tiles;
    A.class_max = (int)class_max;
    A.vec_blocks = (int)std::min<int64_t>(kVecBlocks, (H.ndof + 255) / 256);
    H.cg_terms.ensure(sizeof(double) * terms);
    H.cg_part.ensure(sizeof(double) * ((size_t)nc * tiles + 2 * A.vec_blocks) + sizeof(GridBarrier));
    A.ye = H.cg_terms.as<double>();
    A.part_e = H.cg_part.as<double>();
    A.part_n = A.part_e + (size_t)nc * tiles;
    A.gb = reinterpret_cast<GridBarrier*>(A.part_n + 2 * A.vec_blocks);
    A.s = H.scal.as<KrylovScalars>();
    GG_CUDA(cudaMemsetAsync(A.s, 0, sizeof(KrylovScalars), H.stream));
    if ((dim == 2 ? run<2>(H, A, flight.solves) : run<3>(H, A, flight.solves)) != 0) return 1;
    GG_CUDA(cudaGetLastError());
    H.kernel_launches += 1;
    GG_CUDA(cudaMemcpyAsync(H.h_scal, A.s, sizeof(KrylovScalars), cudaMemcpyDeviceToHost, H.stream));
    GG_CUDA(cudaStreamSynchronize(H.stream));
    if (!H.h_scal->done) {
        H.err = "FP64 CG: grid barrier timed out";
        return GG_ERR_CUDA;
    }
    *iters = H.h_scal->iterations;
    if (H.h_scal->failed == 1) return GG_ERR_NOT_CONVERGED;
    if (H.h_scal->failed) return GG_ERR_NONFINITE;
    return GG_OK;
}

}  // namespace gg
