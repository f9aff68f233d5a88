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
// so an iteration is two barriers.  Small meshes run in one thread-block cluster, whose
// hardware barrier orders the 16 CTAs' global writes in a fraction of a grid barrier;
// larger ones run as a cooperative grid with the counter barrier of gg_grid.cuh.
// Every sum keeps the order of the launches it replaces (gg_solve.cu: 592 blocks of 256
// threads over the vectors, one block per 256-element tile of a class): the partial sums are
// formed per such block, by whichever CTA has it, and added in block index order by every
// CTA, so a solve gives the same bits on every run, for any number of CTAs.  Per iteration:
// 5.2 µs on 32², 7.2 on 64² and 128², 13 on 16³, 19 on 32³, 38 on 48³ (60 as launches).
#include <math.h>

#include <algorithm>
#include <cstring>

#include "gg_grid.cuh"
#include "gg_internal.cuh"
#include "gg_kernels.cuh"
#include "gg_ops.cuh"

namespace gg {

namespace {

constexpr int kVecBlocks = 592;  // blocks of 256 threads the vector sums are split over
constexpr int kCluster = 16;
constexpr int64_t kTermBytes = int64_t(32) << 20;  // element terms that stay in L2

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

template <bool kUseCluster>
__device__ __forceinline__ bool all_sync(GridBarrier* gb, unsigned int* epoch) {
    if constexpr (kUseCluster) {
        (void)gb;
        (void)epoch;
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        return true;
    } else {
        return grid_barrier(gb, epoch);
    }
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

template <int DIM, bool kUseCluster>
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
    if (!all_sync<kUseCluster>(A.gb, &epoch)) return;
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
                en[0] = element_compute<DIM, double, true>(mk, m, M, -1, [&](int c, int a, double v) {
                    __stcg(A.ye + q.term + (int64_t)(a * DIM + c) * A.class_max, v);
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
        if (!all_sync<kUseCluster>(A.gb, &epoch)) return;
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
        if (!all_sync<kUseCluster>(A.gb, &epoch)) return;
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

int cluster_fits(const void* fn, int threads) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(kCluster);
    cfg.blockDim = dim3(threads);
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = kCluster;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, fn, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

template <int DIM>
int run(Handle& H, Cg64Args& A) {
    constexpr int T = cg64_threads<DIM>(), per = T / 256;
    const int work = std::max(A.tiles << DIM, A.vec_blocks);
    const void* fc = (const void*)k_cg64<DIM, true>;
    const void* fg = (const void*)k_cg64<DIM, false>;
    // one cluster while every tile and vector block finds a group of its own in it: 16² / 32² /
    // 48² took 5.9 / 5.2 / 5.5 µs per iteration against 7.4 / 7.0 / 7.6 as a grid; with a
    // second round the 16 SMs lose to the grid (72²: 9.4 against 7.6 µs)
    if (work <= kCluster * per && cluster_fits(fc, T) > 0) {
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(kCluster);
        cfg.blockDim = dim3(T);
        cfg.stream = H.stream;
        cudaLaunchAttribute at{};
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = kCluster;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        GG_CUDA(cudaLaunchKernelEx(&cfg, k_cg64<DIM, true>, A));
        return 0;
    }
    int per_sm = 0;
    GG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fg, T, 0));
    if (per_sm < 1) return 1;
    const int grid = std::min((work + per - 1) / per, per_sm * num_sms());
    GG_CUDA(cudaMemsetAsync(A.gb, 0, sizeof(GridBarrier), H.stream));
    void* args[] = {(void*)&A};
    GG_CUDA(cudaLaunchCooperativeKernel(fg, dim3(grid), dim3(T), args, 0, H.stream));
    return 0;
}

}  // namespace

// x = K⁻¹ b to ‖D⁻¹r‖ ≤ max(rtol‖D⁻¹b‖, 1e-50) in FP64.  Returns 1 when the mesh is outside
// this kernel's limits (element terms beyond kTermBytes, or a class of more tiles than the
// class launches have blocks): the caller then runs the captured launches.
int run_cg64(Handle& H, const double* b, double* x, double rtol, int maxit, int* iters) {
    const int dim = H.dim, nc = 1 << dim;
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
    if ((dim == 2 ? run<2>(H, A) : run<3>(H, A)) != 0) return 1;
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
