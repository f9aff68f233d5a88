// gg_advect.cu -- material point advection on sm_100a.
//
// TimeIntegrand_SecondOrder (StgDomain/Utils/src/TimeIntegrand.cxx:265-335) and the Euler
// update, with _SwarmAdvector_TimeDeriv (PICellerator/MaterialPoints/src/SwarmAdvector.cxx:
// 261-287) as the derivative: locate (the bit-exact search of gg_points.cu), local
// coordinate, Q1 interpolation of the nodal velocity.  A corrector position outside the
// mesh falls back to the first-order update from the start position
// (_TimeIntegrand_RewindToStartAndApplyFirstOrderUpdate, :457-483); a predictor outside
// the mesh is an error (the reference's Journal_Firewall).  Position updates use explicit
// roundings (no FMA contraction), as the x86-64 reference build computes them.
#include "gg_internal.cuh"
#include "gg_kernels.cuh"

namespace gg {

namespace {

constexpr int64_t kPackPoints = 1 << 20;  // points × dim from which the velocities are packed

// kPacked: u holds the components of a node side by side (k_node_velocity), else vector after
// vector
template <int DIM, bool kPacked>
__device__ bool velocity_at(const MeshK& mk, const double* x, const double2* __restrict__ axes,
                            const double* __restrict__ u, double* v) {
    int inds[3] = {0, 0, 0};
#pragma unroll
    for (int d = 0; d < DIM; d++) {
        const double dmax = __dsub_rn(x[d], mk.max[d]);
        if (dmax >= -1e-12 && dmax <= 1e-12) {
            inds[d] = mk.n[d] - 1;
        } else if (x[d] < mk.min[d] || x[d] > mk.max[d]) {
            return false;
        } else {
            const double out = __ddiv_rn(__dsub_rn(x[d], mk.min[d]), mk.sep[d]);
            const double ip = trunc(out);
            const double frac = __dsub_rn(out, ip);
            int i = (int)ip;
            if (i > 0 && frac >= -1e-12 && frac <= 1e-12) i--;
            if (i >= mk.n[d]) i = mk.n[d] - 1;
            inds[d] = i;
        }
    }
    double xi[3] = {0, 0, 0};
    const double2* ax = axes;
#pragma unroll
    for (int d = 0; d < DIM; d++) {
        const double2 g = ax[inds[d]];
        xi[d] = __ddiv_rn(__dsub_rn(x[d], g.x), g.y);
        ax += mk.n[d];
    }
#pragma unroll
    for (int c = 0; c < DIM; c++) v[c] = 0.0;
    const int32_t n0 = inds[0] + mk.nn[0] * (inds[1] + (DIM == 3 ? mk.nn[1] * inds[2] : 0));
#pragma unroll
    for (int a = 0; a < (1 << DIM); a++) {
        double N = (DIM == 2) ? 0.25 : 0.125;
#pragma unroll
        for (int d = 0; d < DIM; d++) N *= 1.0 + (((a >> d) & 1) ? xi[d] : -xi[d]);
        const int32_t n = n0 + (a & 1) + ((a >> 1) & 1) * mk.nn[0] + (DIM == 3 ? ((a >> 2) & 1) * mk.nn[0] * mk.nn[1] : 0);
        double uc[3];
        if constexpr (kPacked) {
            const double2* un = reinterpret_cast<const double2*>(u) + (int64_t)n * (DIM - 1);
            const double2 u01 = un[0];
            uc[0] = u01.x;
            uc[1] = u01.y;
            if (DIM == 3) uc[2] = un[1].x;
        } else {
#pragma unroll
            for (int c = 0; c < DIM; c++) uc[c] = u[(int64_t)c * mk.nnode + n];
        }
#pragma unroll
        for (int c = 0; c < DIM; c++) v[c] += uc[c] * N;
    }
#pragma unroll
    for (int c = 0; c < DIM; c++)
        if (isinf(v[c])) return false;
    return true;
}

// velocity per node, [nnode][2] or [nnode][4], from the component-major vector
template <int DIM>
__global__ void k_node_velocity(int64_t nnode, const double* __restrict__ u, double2* __restrict__ out) {
    for (int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; n < nnode; n += (int64_t)gridDim.x * blockDim.x) {
        out[n * (DIM - 1)] = make_double2(u[n], u[nnode + n]);
        if (DIM == 3) out[n * 2 + 1] = make_double2(u[2 * nnode + n], 0.0);
    }
}

// Bound by the corner velocities: the points are in no spatial order, so every corner is a
// sector of its own.  With the components in separate vectors a 3D stage read 24 of them per
// point; a node's components in one 32-byte sector make it 8 (7.1 M points, two stages:
// 978 → 639 µs).
template <int DIM, bool kPacked>
__global__ void k_advect(MeshK mk, int64_t np, double dt, int order, const double2* __restrict__ axes,
                         const double* __restrict__ u, double* __restrict__ coords, int32_t* __restrict__ flag) {
    const double hdt = __dmul_rn(0.5, dt);
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < np;
         p += (int64_t)gridDim.x * blockDim.x) {
        double x0[3], x[3], k1[3], k2[3];
#pragma unroll
        for (int c = 0; c < DIM; c++) x0[c] = coords[p * DIM + c];
        if (!velocity_at<DIM, kPacked>(mk, x0, axes, u, k1)) {
            atomicAdd(flag, 1);
            continue;
        }
        if (order == 1) {
#pragma unroll
            for (int c = 0; c < DIM; c++) x[c] = __dadd_rn(x0[c], __dmul_rn(dt, k1[c]));
        } else {
#pragma unroll
            for (int c = 0; c < DIM; c++) x[c] = __dadd_rn(x0[c], __dmul_rn(hdt, k1[c]));
            if (velocity_at<DIM, kPacked>(mk, x, axes, u, k2)) {
#pragma unroll
                for (int c = 0; c < DIM; c++) x[c] = __dadd_rn(x0[c], __dmul_rn(dt, k2[c]));
            } else {
#pragma unroll
                for (int c = 0; c < DIM; c++) x[c] = __dadd_rn(x0[c], __dmul_rn(dt, k1[c]));
            }
        }
#pragma unroll
        for (int c = 0; c < DIM; c++) coords[p * DIM + c] = x[c];
    }
}

}  // namespace

int advect(Handle& H, double dt, int order, const double* d_u, double* d_out) {
    (void)d_out;
    H.flag.ensure(sizeof(int32_t) * 4);
    GG_CUDA(cudaMemsetAsync(H.flag.p, 0, sizeof(int32_t) * 4, H.stream));
    const int g = grid_for(H.np, 256);
    const double2* axes = element_axes(H);
    auto move = [&](auto kernel, const void* u) {
        kernel<<<g, 256, 0, H.stream>>>(H.mk, H.np, dt, order, axes, static_cast<const double*>(u), H.coords.as<double>(),
                                        H.flag.as<int32_t>());
    };
    // Packing is a launch of its own, which small swarms do not earn back (µs per call, packed /
    // by component: 64² of 60 50 / 46, 128² of 20 67 / 65, 256×64 of 40 70 / 76, 16³ of 27 58 / 48)
    if (H.np * H.dim < kPackPoints) {
        if (H.dim == 2) move(k_advect<2, false>, d_u);
        else move(k_advect<3, false>, d_u);
    } else {
        H.adv_u.ensure(sizeof(double2) * H.nnode * (H.dim - 1));
        double2* un = H.adv_u.as<double2>();
        const int gn = grid_for(H.nnode, 256);
        if (H.dim == 2) {
            k_node_velocity<2><<<gn, 256, 0, H.stream>>>(H.nnode, d_u, un);
            move(k_advect<2, true>, un);
        } else {
            k_node_velocity<3><<<gn, 256, 0, H.stream>>>(H.nnode, d_u, un);
            move(k_advect<3, true>, un);
        }
    }
    GG_CUDA(cudaGetLastError());
    int32_t bad = 0;
    GG_CUDA(cudaMemcpyAsync(&bad, H.flag.p, sizeof(int32_t), cudaMemcpyDeviceToHost, H.stream));
    GG_CUDA(cudaStreamSynchronize(H.stream));
    H.located = false;
    H.built = false;
    return bad ? GG_ERR_OUT_OF_DOMAIN : GG_OK;
}

}  // namespace gg
