// gg_assembly.cu -- per-point viscosity and PIC quadrature moments on sm_100a.
//
// Replaces, for the Q1-P0 Stokes SLE, the per-element loops of
//   _ConstitutiveMatrixCartesian_AssembleElement (Underworld/Rheology/src/
//       ConstitutiveMatrixCartesian.cxx:206-487) and the rheology chain it runs per point
//       (Rheology_Register_RunRheologies, Rheology_Register.cxx:70-86),
//   _BuoyancyForceTerm_AssembleElement (PICellerator/Utils/src/BuoyancyForceTerm.cxx:414-530),
//   _ThermalBuoyancyForceTerm_AssembleElement (StgFEM/Assembly/src/
//       ThermalBuoyancyForceTerm.cxx:180-235),
//   _UzawaPreconditionerTerm_AssembleElement (StgFEM/SLE/ProvidedSystems/StokesFlow/src/
//       UzawaPreconditionerTerm.cxx:156-239).
//
// On an axis-aligned element B is polynomial in ξ, so K_e = Σ_p c_p Bᵀ D0 B with
// c_p = w_p detJ η_p is fixed by the moments M_m(e) = Σ_p c_p m(ξ_p) of the monomials
// m ∈ {ξ^a η^b ζ^c} that Bᵀ D0 B contains (6 in 2D, 23 in 3D).  One pass over the
// points (sorted by element, in reference order) produces them; the K apply then never
// touches a point again.
//
// Two kernels.  k_points evaluates the rheology chain per point (one thread per point, both
// precisions of a mixed build from the same loads) and leaves the viscosities in point
// order; k_moments sums them per element, four lanes per element, each lane its own
// accumulators over the element's points in order -- the reference's summation order, and
// the same bits whatever the launch shape.  As one kernel (rheology into shared memory, then
// one thread per element with all 39 accumulators) the build held 255 registers, ran 8 warps
// per SM at 0.9 instructions per cycle and took 752 µs (FP64) + 549 µs (FP32) for 7.1 M
// points in 64³ elements; now k_points takes 232 µs for both precisions, k_moments 197 µs
// (FP64) and 111 µs (FP32).
// The element's corner terms of the K diagonal and of the force go to per-element buffers;
// k_gather_corners sums them per node in a fixed element order, so a build gives the same
// bits on every run.
#include <cmath>

#include "gg_internal.cuh"
#include "gg_kernels.cuh"

namespace gg {

namespace {

template <typename R> __device__ __forceinline__ R r_exp(R x);
template <> __device__ __forceinline__ double r_exp<double>(double x) { return exp(x); }
template <> __device__ __forceinline__ float r_exp<float>(float x) { return expf(x); }
template <typename R> __device__ __forceinline__ R r_sqrt(R x);
template <> __device__ __forceinline__ double r_sqrt<double>(double x) { return sqrt(x); }
template <> __device__ __forceinline__ float r_sqrt<float>(float x) { return sqrtf(x); }

// Q1 shape functions at ξ, node order of BilinearElementType/TrilinearElementType.
template <int DIM, typename R>
__device__ __forceinline__ void shape(const R* xi, R* N) {
#pragma unroll
    for (int a = 0; a < (1 << DIM); a++) {
        R v = (DIM == 2) ? R(0.25) : R(0.125);
#pragma unroll
        for (int d = 0; d < DIM; d++) v *= (R(1) + ((a >> d) & 1 ? xi[d] : -xi[d]));
        N[a] = v;
    }
}

// SymmetricTensor_2ndInvariant (StgDomain/Geometry/src/TensorMath.cxx:431-460).
template <int DIM, typename R>
__device__ __forceinline__ R second_invariant(const R* t) {
    if (DIM == 2) return r_sqrt<R>(R(0.5) * (t[0] * t[0] + t[1] * t[1]) + t[2] * t[2]);
    return r_sqrt<R>(R(0.5) * (t[0] * t[0] + t[1] * t[1] + t[2] * t[2]) + t[3] * t[3] +
                     t[4] * t[4] + t[5] * t[5]);
}

struct PointOut {
    double eta, incr;
    uint8_t yielded;
};

// Rheology chain of one material point (RheologyMaterial_RunRheologies).
template <int DIM, typename R>
__device__ PointOut run_rheologies(const MeshK& mk, const gg_material& m, const int* ijk,
                                   int64_t e, const R* xi, const double* __restrict__ T,
                                   const double* __restrict__ pu, const double* __restrict__ pp,
                                   double ep_in, int prev) {
    R eta = R(0);
    R ep = (R)ep_in;
    PointOut out{0.0, 0.0, 0};
    R Tp = R(0);
    bool haveT = false;
    for (int ri = 0; ri < m.n_rheologies; ri++) {
        const gg_rheology& r = m.rheology[ri];
        const int kind = r.kind;
        if (kind == GG_RHEO_MATERIAL_VISCOSITY) {  // MaterialViscosity.cxx:139
            eta = (R)r.eta0;
        } else if (kind == GG_RHEO_ARRHENIUS || kind == GG_RHEO_FRANK_KAMENETSKII) {
            if (!haveT) {
                if (T) {
                    R N[1 << DIM];
                    shape<DIM, R>(xi, N);
                    Tp = R(0);
#pragma unroll
                    for (int a = 0; a < (1 << DIM); a++) Tp += (R)T[elem_node<DIM>(mk, ijk, a)] * N[a];
                }
                haveT = true;
            }
            if (kind == GG_RHEO_FRANK_KAMENETSKII) {  // FrankKamenetskii.cxx:156-160
                eta = (R)r.eta0 * r_exp<R>(-(R)r.theta * Tp);
            } else if (r.activation_volume > (0.0 + 1e-12)) {  // Arrhenius.cxx:200-214
                const R y = (R)(mk.min[1] + (ijk[1] + 0.5) * mk.h[1]) + xi[1] * (R)(0.5 * mk.h[1]);
                const R depth = (R)mk.max[1] - y;
                eta = (R)r.eta0 * r_exp<R>(((R)r.activation_energy + (R)r.activation_volume * depth) /
                                           (Tp + (R)r.reference_temp));
            } else {
                eta = (R)r.eta0 * r_exp<R>((R)r.activation_energy / (Tp + (R)r.reference_temp));
            }
        } else if (kind == GG_RHEO_VON_MISES || kind == GG_RHEO_DRUCKER_PRAGER ||
                   kind == GG_RHEO_BYERLEE) {
            // _YieldRheology_ModifyConstitutiveMatrix (YieldRheology.cxx:190-228)
            if (!prev) continue;
            // strain rate at ξ from the previous velocity: ε̇ = sym(∇u)
            R g[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
#pragma unroll
            for (int a = 0; a < (1 << DIM); a++) {
                const int64_t n = elem_node<DIM>(mk, ijk, a);
                R dN[3];
#pragma unroll
                for (int d = 0; d < DIM; d++) {
                    R v = (R)mk.kappa[d] * (((a >> d) & 1) ? R(1) : R(-1));
#pragma unroll
                    for (int o = 0; o < DIM; o++)
                        if (o != d) v *= (R(1) + (((a >> o) & 1) ? xi[o] : -xi[o]));
                    dN[d] = v;
                }
#pragma unroll
                for (int c = 0; c < DIM; c++) {
                    const R uc = (R)pu[(int64_t)c * mk.nnode + n];
#pragma unroll
                    for (int d = 0; d < DIM; d++) g[c][d] += dN[d] * uc;
                }
            }
            R sr[6], st[6];
            if (DIM == 2) {
                sr[0] = g[0][0]; sr[1] = g[1][1]; sr[2] = R(0.5) * (g[0][1] + g[1][0]);
            } else {
                sr[0] = g[0][0]; sr[1] = g[1][1]; sr[2] = g[2][2];
                sr[3] = R(0.5) * (g[0][1] + g[1][0]);
                sr[4] = R(0.5) * (g[0][2] + g[2][0]);
                sr[5] = R(0.5) * (g[1][2] + g[2][1]);
            }
            const int ns = DIM == 2 ? 3 : 6;
            R trs = R(0), trsr = R(0);
            for (int k = 0; k < ns; k++) st[k] = R(2) * eta * sr[k];  // isotropic D·ε̇
            for (int k = 0; k < DIM; k++) { trs += st[k]; trsr += sr[k]; }
            for (int k = 0; k < DIM; k++) { sr[k] -= trsr / R(DIM); st[k] -= trs / R(DIM); }
            const R sr_ii = second_invariant<DIM, R>(sr);
            const R ind = second_invariant<DIM, R>(st);  // _VonMises_GetYieldIndicator
            // StrainWeakening_CalcRatio (StrainWeakening.cxx:497-519)
            R ratio = R(0);
            const bool sw = m.has_strain_weakening && r.strain_weakening;
            if (sw) {
                if (ep < R(0)) ep = R(0);
                ratio = (ep - (R)m.strain_weakening.initial_softening_strain) /
                        ((R)m.strain_weakening.final_softening_strain -
                         (R)m.strain_weakening.initial_softening_strain);
                if (ratio > R(1)) ratio = R(1);
                if (ratio < R(0)) ratio = R(0);
            }
            R crit;
            if (kind == GG_RHEO_VON_MISES) {  // VonMises.cxx:183-204
                crit = (R)r.cohesion * (R(1) - ratio) + (R)r.cohesion_after_softening * ratio;
            } else if (kind == GG_RHEO_DRUCKER_PRAGER) {  // DruckerPrager.cxx:296-412
                const R pressure = pp ? (R)pp[e] : R(0);
                // elements along a flagged wall take the boundary strength (:341-361)
                const int bw = r.boundary_walls;
                const bool inb = ((bw & 1) && ijk[0] == 0) || ((bw & 2) && ijk[0] == mk.n[0] - 1) ||
                                 ((bw & 4) && ijk[1] == 0) || ((bw & 8) && ijk[1] == mk.n[1] - 1) ||
                                 (DIM == 3 && (((bw & 16) && ijk[2] == 0) || ((bw & 32) && ijk[2] == mk.n[2] - 1)));
                const R mu = inb ? (R)r.boundary_friction_coefficient * (R(1) - ratio) +
                                       (R)r.boundary_friction_coefficient_after_softening * ratio
                                 : (R)r.friction_coefficient * (R(1) - ratio) +
                                       (R)r.friction_coefficient_after_softening * ratio;
                const R C = inb ? (R)r.boundary_cohesion * (R(1) - ratio) + (R)r.boundary_cohesion_after_softening * ratio
                                : (R)r.cohesion * (R(1) - ratio) + (R)r.cohesion_after_softening * ratio;
                R factor, fs;
                if (DIM == 2) {
                    factor = R(1) / r_sqrt<R>(R(1) + mu * mu);
                    fs = mu * pressure * factor + C * factor;
                } else {
                    const R cphi = R(1) / r_sqrt<R>(R(1) + mu * mu), sphi = mu * cphi;
                    factor = R(2) * cphi / (r_sqrt<R>(R(3)) * (R(3) - sphi));
                    fs = mu * factor * pressure + C * R(3) * factor;
                }
                R mys = (R)r.minimum_yield_stress;
                if (mys == R(0)) mys = C;
                if (fs < mys * factor) fs = mys * factor;
                crit = fs;
            } else {  // Byerlee.cxx:163-187
                const R y = (R)(mk.min[1] + (ijk[1] + 0.5) * mk.h[1]) + xi[1] * (R)(0.5 * mk.h[1]);
                crit = (R)r.cohesion + (R)r.depth_coefficient * ((R)mk.max[1] - y);
            }
            if (sw) {  // _StrainWeakening_CalcIncrementIsotropic (StrainWeakening.cxx:470-495)
                R beta = R(1) - crit / ind;
                if (beta < R(0)) beta = R(0);
                out.incr = (double)((crit / eta) *
                                    (beta / (R(1) - beta) - (R)m.strain_weakening.healing_rate * ep));
            }
            if (crit < ind) {
                out.yielded = 1;
                if (kind == GG_RHEO_DRUCKER_PRAGER) {  // DruckerPrager.cxx:414-446
                    R v = (r.max_strain_rate > 0 && sr_ii > (R)r.max_strain_rate)
                              ? crit / (R(2) * (R)r.max_strain_rate)
                              : crit / (R(2) * sr_ii);
                    if (v < (R)r.minimum_viscosity) v = (R)r.minimum_viscosity;
                    eta = v;
                } else if (r.strain_rate_softening) {  // VonMises.cxx:258-263
                    eta = R(2) * crit * crit * eta / (crit * crit + ind * ind);
                } else {  // VonMises.cxx:264-271
                    const R beta = R(1) - crit / ind;
                    R corr = -eta * beta;
                    if ((eta + corr) < (R)r.minimum_viscosity) corr = (R)r.minimum_viscosity - eta;
                    eta += corr;
                }
            }
        }
    }
    out.eta = (double)eta;
    return out;
}

// Per point: viscosity in FP64, with kBoth also by the FP32 rheology chain, and the
// temperature where a force term reads it (temp null: none does; T null: it is 0).
// Bound by its loads and stores (60-90 bytes per point) once enough warps cover the
// exponential's latency: at 255 registers, one block per SM, it took 651 µs for 7.1 M points;
// three blocks spill a little in the yield laws and take 232 (two took 3 % more), 32-bit element
// indices in both.
template <int DIM, bool kBoth>
__global__ void __launch_bounds__(256, 3)
k_points(MeshK mk, int64_t np, const int32_t* __restrict__ cell_s, const double* __restrict__ xi_s,
         const int32_t* __restrict__ mat_s, const double* __restrict__ ps_s, const double* __restrict__ T,
         const double* __restrict__ pu, const double* __restrict__ pp, int prev, double rayleigh,
         const gg_material* __restrict__ materials, float* __restrict__ eta32, double* __restrict__ temp,
         double* __restrict__ eta_s, double* __restrict__ incr_s, uint8_t* __restrict__ yld_s) {
    constexpr int NEN = 1 << DIM;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < np; i += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t pe = (uint32_t)cell_s[i], row = pe / (uint32_t)mk.n[0];
        const int ijk[3] = {(int)(pe - row * (uint32_t)mk.n[0]), (int)(row % (uint32_t)mk.n[1]),
                            (int)(row / (uint32_t)mk.n[1])};
        double xi[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int d = 0; d < DIM; d++) xi[d] = xi_s[(int64_t)d * np + i];
        const gg_material& m = materials[mat_s[i]];
        const double ps = ps_s[i];
        const PointOut po = run_rheologies<DIM, double>(mk, m, ijk, pe, xi, T, pu, pp, ps, prev);
        eta_s[i] = po.eta;
        incr_s[i] = po.incr;
        yld_s[i] = po.yielded;
        if (kBoth) {
            float x32[3] = {0.f, 0.f, 0.f};
#pragma unroll
            for (int d = 0; d < DIM; d++) x32[d] = (float)xi[d];
            eta32[i] = (float)run_rheologies<DIM, float>(mk, m, ijk, pe, x32, T, pu, pp, ps, prev).eta;
        }
        if (temp) {
            double Tp = 0.0;
            if (T && (rayleigh != 0.0 || m.alpha != 0.0)) {
                double N[NEN];
                shape<DIM, double>(xi, N);
#pragma unroll
                for (int a = 0; a < NEN; a++) Tp += T[elem_node<DIM>(mk, ijk, a)] * N[a];
            }
            temp[i] = Tp;
        }
    }
}

// Per element, four lanes, over its points in order: c_p = w_p detJ η_p and the force weights
// φ_p = detJ w ρ g, ψ_p = detJ w Ra T are formed on the way; lane q < 3 sums the moments of
// ξ-exponent q (every lane the same instructions, with its own power of ξ), lane q the force
// terms of corners q·NC ….  want_phi 0 / temp null: those weights are zero for every point.
// Then every lane takes all moments and forms its corners' diagonal terms.
// Eight elements per warp keep an SM at 20 (FP64, 3D) to 36 warps, where one thread per element
// and 39 accumulators left 8; the eight streams of points of a warp meet in L1.  Bound by those
// loads: 48 % of the issue slots, 25 % of the DRAM peak (deeper unrolling changed nothing).
template <int DIM, typename R, bool kForce>
__global__ void __launch_bounds__(128)
k_moments(MeshK mk, int64_t nel, const int32_t* __restrict__ offsets, const double* __restrict__ xi_s, int64_t np,
          const R* __restrict__ eta, const double* __restrict__ w_s, const int32_t* __restrict__ mat_s,
          const double* __restrict__ temp, const gg_material* __restrict__ materials, int want_phi, double gravity,
          double rayleigh, R* __restrict__ mom, R* __restrict__ kcorner, double* __restrict__ sdiag,
          double* __restrict__ fcorner, int32_t* __restrict__ flag) {
    constexpr unsigned kFull = 0xffffffffu;
    constexpr int NM = n_moments<DIM>(), NEN = 1 << DIM, NC = NEN / 4, NZ = DIM == 3 ? 3 : 1;
    const int q = threadIdx.x & 3;
    const int64_t e = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 2;
    const bool own = e < nel;
    const int32_t b = own ? offsets[e] : 0, en = own ? offsets[e + 1] : 0;
    // _ConstantWeights_Calculate, or the per-point weight (DVCWeights)
    const double wconst = (double)(1 << DIM) / (double)(en - b);
    R acc[3][NZ];
#pragma unroll
    for (int bb = 0; bb < 3; bb++)
#pragma unroll
        for (int cc = 0; cc < NZ; cc++) acc[bb][cc] = R(0);
    double F[NC], Psi[NC];
#pragma unroll
    for (int j = 0; j < NC; j++) { F[j] = 0.0; Psi[j] = 0.0; }
#pragma unroll 4
    for (int32_t i = b; i < en; i++) {
        const double xd = xi_s[i], yd = xi_s[np + i], zd = DIM == 3 ? xi_s[2 * np + i] : 0.0;
        const double w = w_s ? w_s[i] : wconst;
        const R c = (R)(w * mk.detJ) * eta[i], x = (R)xd, y = (R)yd, z = (R)zd;
        const R px = q == 0 ? R(1) : q == 1 ? x : x * x;
        const R pxy[3] = {px, px * y, px * (y * y)};
        const R zz = z * z;
#pragma unroll
        for (int bb = 0; bb < 3; bb++) {
            acc[bb][0] += c * pxy[bb];
            if (DIM == 3) {
                acc[bb][NZ == 3 ? 1 : 0] += c * (pxy[bb] * z);
                acc[bb][NZ == 3 ? 2 : 0] += c * (pxy[bb] * zz);
            }
        }
        if (kForce) {
            const double Tp = temp ? temp[i] : 0.0;
            double ph = 0.0;
            if (want_phi) {
                const gg_material& m = materials[mat_s[i]];
                const double rho = m.density * (1.0 - m.alpha * Tp);
                ph = mk.detJ * w * rho * gravity;
            }
            const double ps = temp ? mk.detJ * w * (rayleigh * Tp) : 0.0;
#pragma unroll
            for (int j = 0; j < NC; j++) {
                const int a = q * NC + j;
                double N = DIM == 2 ? 0.25 : 0.125;
                N *= 1.0 + ((a & 1) ? xd : -xd);
                N *= 1.0 + ((a & 2) ? yd : -yd);
                if (DIM == 3) N *= 1.0 + ((a & 4) ? zd : -zd);
                F[j] += ph * N;
                Psi[j] += ps * N;
            }
        }
    }
    if (own && q == 0 && en == b) atomicAdd(flag, 1);  // empty element
    R M[NM];
#pragma unroll
    for (int aa = 0; aa < 3; aa++)
#pragma unroll
        for (int bb = 0; bb < 3; bb++)
#pragma unroll
            for (int cc = 0; cc < NZ; cc++) {
                const int slot = mom_slot<DIM>(aa, bb, cc);
                if (slot >= 0) M[slot] = __shfl_sync(kFull, acc[bb][cc], aa, 4);
            }
    if (own) {
#pragma unroll
        for (int m = 0; m < NM; m++)
            if ((m & 3) == q) mom[(int64_t)m * nel + e] = M[m];
    }
    // element diagonal of K from the moments:
    // K[(a,c),(a,c)] = Σ_p c_p [ Σ_d (∂N_a/∂x_d)² + (∂N_a/∂x_c)² ]
    double ratio[NC][DIM], G[NC][DIM];  // G_e / K_e diagonal and G_e of this lane's dofs
#pragma unroll
    for (int j = 0; j < NC; j++) {
        const int a = q * NC + j;
        double sg[3];
#pragma unroll
        for (int o = 0; o < 3; o++) sg[o] = ((a >> o) & 1) ? 1.0 : -1.0;
        double S[3];
#pragma unroll
        for (int d = 0; d < DIM; d++) {
            // Σ_p c_p Π_{o≠d} (1 + s_o ξ_o)²,  (1+sξ)² = 1 + 2sξ + ξ²
            double v = 0.0;
#pragma unroll
            for (int k0 = 0; k0 < 3; k0++)
#pragma unroll
                for (int k1 = 0; k1 < 3; k1++)
#pragma unroll
                    for (int k2 = 0; k2 < 3; k2++) {
                        const int ex[3] = {k0, k1, k2};
                        bool ok = true;
                        double coef = 1.0;
#pragma unroll
                        for (int o = 0; o < 3; o++) {
                            if (o >= DIM || o == d) { if (ex[o] != 0) ok = false; continue; }
                            coef *= ex[o] == 1 ? 2.0 * sg[o] : 1.0;
                        }
                        if (!ok) continue;
                        v += coef * (double)M[mom_slot<DIM>(k0, k1, k2)];
                    }
            S[d] = v * mk.kappa[d] * mk.kappa[d];
        }
        double tot = 0.0;
#pragma unroll
        for (int d = 0; d < DIM; d++) tot += S[d];
#pragma unroll
        for (int c = 0; c < DIM; c++) {
            const double dg = tot + S[c];
            if (own) kcorner[(int64_t)(a * DIM + c) * nel + e] = (R)dg;
            if (kForce) {
                G[j][c] = mk.Ge[a][c];
                ratio[j][c] = G[j][c] / dg;
            }
        }
        if (kForce && own) {
            fcorner[(int64_t)a * nel + e] = F[j];
            fcorner[(int64_t)(NEN + a) * nel + e] = Psi[j];
        }
    }
    if (kForce) {
        // Ĝ_e = Σ G_e² / K_e diagonal, over every dof (UzawaPreconditionerTerm.cxx:199-215), in
        // dof order: the running sum passes from lane to lane
        double sd = 0.0;
#pragma unroll
        for (int l = 0; l < 4; l++) {
            double s = sd;
#pragma unroll
            for (int j = 0; j < NC; j++)
#pragma unroll
                for (int c = 0; c < DIM; c++) s += G[j][c] * ratio[j][c];
            sd = __shfl_sync(kFull, s, l, 4);
        }
        if (own && q == 0) sdiag[e] = sd;
    }
}

// Node sums of the element corner terms in a fixed element order (corner a' = 0 … 2^dim−1
// of the node in its adjacent elements), so the assembled diagonal and force vector are
// the same bits on every run: kdiag[c][n] = Σ_e K_e[(a',c),(a',c)],
// f[c][n] = Σ_e (g_c F_e[a'] + [c = y] Ψ_e[a']).
template <int DIM, typename R>
__global__ void k_gather_corners(MeshK mk, const R* __restrict__ kcorner, const double* __restrict__ fcorner,
                                 double g0, double g1, double g2, R* __restrict__ kdiag, double* __restrict__ f) {
    constexpr int NEN = 1 << DIM;
    const int64_t nnode = mk.nnode, nel = mk.nel;
    for (int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; n < nnode; n += (int64_t)gridDim.x * blockDim.x) {
        const int i = (int)(n % mk.nn[0]);
        const int j = (int)((n / mk.nn[0]) % mk.nn[1]);
        const int k = DIM == 3 ? (int)(n / ((int64_t)mk.nn[0] * mk.nn[1])) : 0;
        R kd[DIM];
        double fv[DIM];
#pragma unroll
        for (int c = 0; c < DIM; c++) { kd[c] = R(0); fv[c] = 0.0; }
#pragma unroll
        for (int a = 0; a < NEN; a++) {
            const int ei = i - (a & 1), ej = j - ((a >> 1) & 1), ek = DIM == 3 ? k - ((a >> 2) & 1) : 0;
            if (ei < 0 || ej < 0 || ek < 0 || ei >= mk.n[0] || ej >= mk.n[1] || (DIM == 3 && ek >= mk.n[2])) continue;
            const int64_t e = ei + (int64_t)mk.n[0] * (ej + (int64_t)mk.n[1] * ek);
#pragma unroll
            for (int c = 0; c < DIM; c++) kd[c] += kcorner[(int64_t)(a * DIM + c) * nel + e];
            if (f) {
                const double Fa = fcorner[(int64_t)a * nel + e], Pa = fcorner[(int64_t)(NEN + a) * nel + e];
#pragma unroll
                for (int c = 0; c < DIM; c++) {
                    double v = (c == 0 ? g0 : (c == 1 ? g1 : g2)) * Fa;
                    if (c == 1) v += Pa;
                    fv[c] += v;
                }
            }
        }
#pragma unroll
        for (int c = 0; c < DIM; c++) {
            kdiag[(int64_t)c * nnode + n] = kd[c];
            if (f) f[(int64_t)c * nnode + n] = fv[c];
        }
    }
}

}  // namespace

// The material table lives in a per-handle device buffer, so concurrent handles (threads,
// streams) never share it.
void upload_materials(Handle& H) {
    H.d_materials.ensure(sizeof(gg_material) * GG_MAX_MATERIALS);
    H.h_materials.assign(H.materials.begin(), H.materials.end());
    GG_CUDA(cudaMemcpyAsync(H.d_materials.p, H.h_materials.data(), sizeof(gg_material) * H.h_materials.size(),
                            cudaMemcpyHostToDevice, H.stream));
}

// kdiag (and f) from the corner terms of the last build launch
template <int DIM, typename R>
static void gather_corners(Handle& H, R* kdiag, double* f) {
    double g[3] = {H.force.g_hat[0], H.force.g_hat[1], H.force.g_hat[2]};
    const double* fc = f ? H.fcorner.as<double>() : nullptr;
    k_gather_corners<DIM, R><<<grid_for(H.nnode, 256), 256, 0, H.stream>>>(
        H.mk, reinterpret_cast<const R*>(H.kcorner.p), fc, g[0], g[1], g[2], kdiag, f);
    GG_CUDA(cudaGetLastError());
}

// Whether the force weights of a build can be anything but zero.  A zero gravity or Rayleigh
// number, or a temperature that is not set (0), makes them zero unless the factor beside it is
// not finite: a density, a thermal expansivity (through it the temperature) or the Rayleigh
// number.  Those weights are NaN, and so are the force and the solve that reads it.
static bool any_alpha(const Handle& H) {
    for (const gg_material& m : H.materials)
        if (H.has_T ? m.alpha != 0.0 : !std::isfinite(m.alpha)) return true;
    return false;
}
static bool phi_nonzero(const Handle& H) {
    if (H.force.gravity != 0.0 || any_alpha(H)) return true;
    for (const gg_material& m : H.materials)
        if (!std::isfinite(m.density)) return true;
    return false;
}
static bool psi_nonzero(const Handle& H) {
    return !std::isfinite(H.force.rayleigh) || (H.has_T && (H.force.rayleigh != 0.0 || any_alpha(H)));
}

template <int DIM>
static void launch_build(Handle& H, bool mixed, int prev, const double* pu, const double* pp) {
    const int64_t np = H.np_in, nel = H.nel;
    cudaStream_t st = H.stream;
    const double* T = H.has_T ? H.T.as<double>() : nullptr;
    const double* w = H.weights.mode == GG_WEIGHTS_DVC && H.dvc_valid ? H.w_s.as<double>() : nullptr;
    double* temp = psi_nonzero(H) ? H.pt_temp.as<double>() : nullptr;
    // the points' elements in input order are not read again after gg_locate: their words
    // hold the FP32 viscosities
    float* eta32 = mixed ? H.cell.as<float>() : nullptr;
    auto points = [&](auto kernel) {
        kernel<<<grid_for(np, 256), 256, 0, st>>>(H.mk, np, H.cell_s.as<int32_t>(), H.xi_s.as<double>(),
                                                  H.mat_s.as<int32_t>(), H.ps_s.as<double>(), T, pu, pp, prev,
                                                  H.force.rayleigh, H.d_materials.as<gg_material>(), eta32, temp,
                                                  H.eta_s.as<double>(), H.incr_s.as<double>(), H.yld_s.as<uint8_t>());
        GG_CUDA(cudaGetLastError());
    };
    if (mixed) points(k_points<DIM, true>);
    else points(k_points<DIM, false>);
    const unsigned grid = (unsigned)((4 * nel + 127) / 128);
    k_moments<DIM, double, true><<<grid, 128, 0, st>>>(
        H.mk, nel, H.offsets.as<int32_t>(), H.xi_s.as<double>(), np, H.eta_s.as<double>(), w, H.mat_s.as<int32_t>(),
        temp, H.d_materials.as<gg_material>(), phi_nonzero(H), H.force.gravity, H.force.rayleigh, H.mom64.as<double>(),
        H.kcorner.as<double>(), H.sdiag.as<double>(), H.fcorner.as<double>(), H.flag.as<int32_t>());
    GG_CUDA(cudaGetLastError());
    gather_corners<DIM, double>(H, H.kdiag64.as<double>(), H.f.as<double>());
    if (mixed) {
        k_moments<DIM, float, false><<<grid, 128, 0, st>>>(
            H.mk, nel, H.offsets.as<int32_t>(), H.xi_s.as<double>(), np, eta32, w, nullptr, nullptr, nullptr, 0, 0.0, 0.0,
            H.mom32.as<float>(), H.kcorner.as<float>(), nullptr, nullptr, H.flag.as<int32_t>());
        GG_CUDA(cudaGetLastError());
        gather_corners<DIM, float>(H, H.kdiag32.as<float>(), nullptr);
    }
}

int build_operator(Handle& H, int precision, int prev, const double* d_prev_u,
                   const double* d_prev_p) {
    cudaStream_t st = H.stream;
    const int64_t nel = H.nel, nd = H.ndof;
    const int nm = H.nm;
    H.mom64.ensure(sizeof(double) * nm * nel);
    H.kdiag64.ensure(sizeof(double) * nd);
    H.sdiag.ensure(sizeof(double) * nel);
    H.f.ensure(sizeof(double) * nd);
    H.flag.ensure(sizeof(int32_t) * 4);
    // element corner terms of the diagonal and the force, summed per node after the build
    const int nen = 1 << H.dim;
    H.kcorner.ensure(sizeof(double) * nen * H.dim * nel);
    H.fcorner.ensure(sizeof(double) * 2 * nen * nel);
    upload_materials(H);
    GG_CUDA(cudaMemsetAsync(H.flag.p, 0, sizeof(int32_t) * 4, st));
    const bool mixed = precision == GG_PRECISION_MIXED;
    if (psi_nonzero(H)) H.pt_temp.ensure(sizeof(double) * H.np_in);
    if (mixed) {
        H.mom32.ensure(sizeof(float) * nm * nel);
        H.kdiag32.ensure(sizeof(float) * nd);
    }
    if (H.dim == 2) launch_build<2>(H, mixed, prev, d_prev_u, d_prev_p);
    else launch_build<3>(H, mixed, prev, d_prev_u, d_prev_p);
    int32_t empty = 0;
    GG_CUDA(cudaMemcpyAsync(&empty, H.flag.p, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
    GG_CUDA(cudaStreamSynchronize(st));
    if (empty) return GG_ERR_EMPTY_CELL;
    return GG_OK;
}

}  // namespace gg
