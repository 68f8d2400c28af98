// Mixed-precision pair passes: pair geometry and table evaluation in FP32, in angstrom and
// eV, with every sum over pairs (per-atom densities, forces and energies, the virial, Born
// stress, Born tensor and Laplacian) accumulated in FP64 and converted to cgs at the end;
// the per-atom helpers g_i and h_i of the density pass are summed in FP32 along the row.
//
// Pair forces stay exactly antisymmetric: dp_ij = -dp_ji bit for bit (IEEE subtraction and
// round-to-nearest-even are odd functions), every other pair quantity depends on r only,
// and the two EAM cross terms of dE/dr are rounded separately and added commutatively.
// With the per-atom sums in FP64 the total momentum is conserved as in the FP64 path.
//
// The neighbour list, the embedding function and the integrator are shared with the FP64
// path (FP64, cgs): the list comes from the FP64 coordinates, and k_kick_drift refreshes
// the FP32 positions posf after every drift.
#include "kernels.cuh"
#include "pair_common.cuh"

namespace mdelast {

namespace {

// interval index, at most n - 1, and local coordinate; x >= 0
__device__ __forceinline__ int tab_locate_f(float x, float inv_h, int n, float &t) {
    float const u = __fmul_rn(x, inv_h);
    int const i = min(__float2int_rz(u), n - 1);
    t = __fsub_rn(u, __int2float_rn(i));
    return i;
}

// Quintic records (8 floats, TablesView::rrf: c0..c5, 3 c3, 5 c5) and derivative records
// (rdf: c1, 2 c2, 3 c3, 4 c4, 5 c5, 6 c3, 12 c4, 20 c5). The pair force is evaluated from
// both of its atoms, in different code paths of the force pass; its arithmetic is written with
// explicit rounding (no contraction left to the compiler) so that both evaluations, and those
// from the staged tables, give the same bits.
__device__ __forceinline__ float horner4(float t, float a, float b, float c, float d) {
    return __fmaf_rn(t, __fmaf_rn(t, __fmaf_rn(t, d, c), b), a);
}
__device__ __forceinline__ float tabf_v(const float *c, float t) {
    return __fmaf_rn(t, __fmaf_rn(t, horner4(t, c[2], c[3], c[4], c[5]), c[1]), c[0]);
}
__device__ __forceinline__ float tabf_d1(const float *c, float t, float inv_h) {
    return __fmul_rn(__fmaf_rn(t, horner4(t, __fmul_rn(2.f, c[2]), c[6], __fmul_rn(4.f, c[4]), c[7]),
                               c[1]), inv_h);
}
__device__ __forceinline__ float tabf_d2(const float *c, float t, float inv_h2) {
    return __fmul_rn(horner4(t, __fmul_rn(2.f, c[2]), __fmul_rn(2.f, c[6]), __fmul_rn(12.f, c[4]),
                             __fmul_rn(4.f, c[7])), inv_h2);
}
__device__ __forceinline__ float tabd_d1(const float *d, float t, float inv_h) {
    return __fmul_rn(__fmaf_rn(t, horner4(t, d[1], d[2], d[3], d[4]), d[0]), inv_h);
}
__device__ __forceinline__ float tabd_d2(const float *d, float t, float inv_h2) {
    return __fmul_rn(horner4(t, d[1], d[5], d[6], d[7]), inv_h2);
}
// the derivative record of the coefficients c0..c5, as the host rounds it
__device__ __forceinline__ void derivative_record(const float *c, float (&d)[8]) {
    d[0] = c[1];
    d[1] = __fmul_rn(2.f, c[2]);
    d[2] = __fmul_rn(3.f, c[3]);
    d[3] = __fmul_rn(4.f, c[4]);
    d[4] = __fmul_rn(5.f, c[5]);
    d[5] = __fmul_rn(6.f, c[3]);
    d[6] = __fmul_rn(12.f, c[4]);
    d[7] = __fmul_rn(20.f, c[5]);
}

// FP32 counterpart of tab_eval (device.cuh): QUINTIC interval data are the 6 quintic
// coefficients, BSPLINE data three cubics (values of the splines of f, f', f''); both with
// explicit rounding.
__device__ __forceinline__ float cubicf_at(const float *p, float t) {
    float4 const a = __ldg(reinterpret_cast<const float4 *>(p));
    return __fmaf_rn(t, __fmaf_rn(t, __fmaf_rn(t, a.w, a.z), a.y), a.x);
}

template <int IP, bool NV, bool ND1, bool ND2>
__device__ __forceinline__ void tabf_eval(const float *p, float t, float inv_h, float inv_h2,
                                          float &v, float &d1, float &d2) {
    if constexpr (IP == MDELAST_BSPLINE) {
        if (NV)
            v = cubicf_at(p, t);
        if (ND1)
            d1 = cubicf_at(p + 4, t);
        if (ND2)
            d2 = cubicf_at(p + 8, t);
    } else {
        float c[8];
        ld256(p, c);
        if (NV)
            v = tabf_v(c, t);
        if (ND1)
            d1 = tabf_d1(c, t, inv_h);
        if (ND2)
            d2 = tabf_d2(c, t, inv_h2);
    }
}

} // namespace

// FP32 wrapped positions of every atom from the FP64 coordinates and the current box.
__global__ void k_posf(AtomsView A) {
    int const i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= A.n_pad)
        return;
    int const r = A.rep_of[i];
    if (r >= 0)
        A.posf[i] = position_f(A.crd[i], A.rep + r);
}

// One lane's share of an atom row in the density pass: branch-free body, three entries per
// unrolled pass (two spilled at 8 blocks per SM: 0.187 against 0.167 ms at 16 x 13,500 atoms); an entry beyond the cutoff adds zeros. UC: every
// density cutoff is at least the pair cutoff (no per-type test).
template <bool OBS, int TPA, int IP, typename IX, bool UC>
__device__ __forceinline__ void dens_loop(AtomsView const &A, TablesView const &T, float4 pi,
                                          float3 L, float3 iL, PairRow<IX> const &row, int nu,
                                          int ntot, int sub, double &rho, float (&g)[6], float (&hv)[3]) {
    // the next partner's record and the list entry after it are loaded ahead, so the
    // entry's load does not delay the record's
    float4 pn = A.posf[sub < ntot ? row.at(list_slot(sub, nu, A.pmaxn)) : row.base];
    int jn = sub < ntot ? row.at(list_slot(min(sub + TPA, ntot - 1), nu, A.pmaxn)) : row.base;
#pragma unroll 3
    for (int kk = sub; kk < ntot; kk += TPA) {
        float4 const pj = pn;
        pn = A.posf[jn];
        jn = row.at(list_slot(min(kk + 2 * TPA, ntot - 1), nu, A.pmaxn));
        float dx, dy, dz;
        float const r2 = min_image_f(pi, pj, L, iL, dx, dy, dz);
        float const idr = rsqrtf(r2);
        float const dr = __fmul_rn(r2, idr);
        int const tj = __float_as_int(pj.w);
        bool const in_cut = !(r2 > T.fr_cut_sq) && (UC || !(dr > T.feam_rcut[tj]));
        float t;
        int const k = tab_locate_f(dr, T.finv_hr, T.nri, t);
        float v = 0.f, d1 = 0.f, d2 = 0.f;
        tabf_eval<IP, true, OBS, false>(
            T.rrf + static_cast<unsigned>(tj * T.nri + k) * TabFmt<IP>::kFf, t, T.finv_hr,
            T.finv_hr2, v, d1, d2);
        if (!in_cut) {
            v = 0.f;
            d1 = 0.f;
        }
        rho += static_cast<double>(v);
        if (OBS) {
            float const ar = d1 * idr;
            float const ap[3] = {ar * dx, ar * dy, ar * dz};
            g[0] += ap[0] * dx;
            g[1] += ap[1] * dy;
            g[2] += ap[2] * dz;
            g[3] += ap[1] * dz;
            g[4] += ap[0] * dz;
            g[5] += ap[0] * dy;
            hv[0] += ap[0];
            hv[1] += ap[1];
            hv[2] += ap[2];
        }
    }
}

// Density pass of md_driver.cpp:195-277 in mixed precision (see k_density for the roles).
// The atom's terms of the block's FP64 sums (embedding energy, the per-atom Born term
// F''_i g_i g_i^T and the Laplacian term) are formed in every lane of the atom, so that
// warp_slots spreads them over the lanes with 7 exchanges at 4 lanes per atom; each lane
// carries one running sum. (Before, 23 warp sums per atom group: 18 % of the pass's L1 data
// pipe went to their shuffles.)
//
// Bounded to 8 blocks of 128 threads per SM (64 registers; the compiler's own choice is 72,
// 7 blocks): a few bytes of spills, and the extra warps hide more of the gather latency
// (0.194 -> 0.182 ms at 16 x 13,500 atoms; 9 and 10 blocks spilled more and ran slower).
// Bound by the L1 data pipe (65 % of its wavefront rate, issue 49 %): at 16 x 13,500 atoms and
// 4 lanes per atom 0.195 -> 0.162 ms with the 32-byte records and warp_slots.
template <bool OBS, int TPA, int IP, typename IX>
__global__ void __launch_bounds__(kBlock, 8) k_density_mx(AtomsView A, TablesView T) {
    chain_begin();
    if (halted(A)) // a list build ran out of capacity: nothing until the host regrows
        return;
    constexpr int kF = TabFmt<IP>::kF;
    constexpr int kSlots = OBS ? D_NSUM : 1, kP2 = slots_pow2(kSlots);
    double acc = 0.; // the block sum of this lane's slot over the warp's atom groups
    int const r = A.dblk_rep[blockIdx.x];
    Replica const *R = A.rep + r;
    int const lb = blockIdx.x - R->dblk_begin, nb = R->dblk_n;
    int const apb = kBlock / TPA, sub = threadIdx.x % TPA;
    int const n_slots = R->n_blocks * kBlock;
    float3 L, iL;
    box_f(R, L, iL);
    double const a3 = kAng * kAng * kAng;
    for (int a0 = lb * apb; a0 < n_slots; a0 += nb * apb) {
        int const a = a0 + static_cast<int>(threadIdx.x) / TPA;
        int const i = R->atom_begin + a;
        bool const valid = a < R->n_atoms && T.has_eam;
        double rho = 0.;
        float g[6] = {0, 0, 0, 0, 0, 0}, hv[3] = {0, 0, 0};
        int ti = 0;
        if (valid) {
            float4 const pi = A.posf[i];
            ti = __float_as_int(pi.w);
            int const nu = A.pn_up[i], ntot = nu + A.pn_dn[i];
            PairRow<IX> const row = pair_row<IX>(A, i, R->atom_begin);
            // uniform cutoffs (every setfl potential): no per-function cutoff test
            if (T.fuc)
                dens_loop<OBS, TPA, IP, IX, true>(A, T, pi, L, iL, row, nu, ntot, sub, rho, g,
                                                  hv);
            else
                dens_loop<OBS, TPA, IP, IX, false>(A, T, pi, L, iL, row, nu, ntot, sub, rho, g,
                                                  hv);
        }
        rho = group_sum<TPA>(rho);
        if (OBS) {
#pragma unroll
            for (int u = 0; u < 6; ++u)
                g[u] = group_sum<TPA>(g[u]);
#pragma unroll
            for (int u = 0; u < 3; ++u)
                hv[u] = group_sum<TPA>(hv[u]);
        }
        double F = 0., d2F = 0.;
        if (valid) { // every lane of the atom, stored by the first
            // the embedding function in FP64 and cgs (eam.hpp:48-70)
            double const rc = rho / a3;
            if (rc > T.rhomax[ti])
                status_or(A.rep + r, MDELAST_FATAL_RHO_MAX);
            double t;
            int const k = tab_locate(rc, T.inv_hf, T.nfi, t);
            double dF = 0.;
            tab_eval<IP, true, true, OBS>(T.Ft + (static_cast<size_t>(ti) * T.nfi + k) * kF, t,
                                          T.inv_hf, T.inv_hf2, F, dF, d2F);
            // F' [erg cm^3] -> [eV A^3] and F'' [erg cm^6] -> [eV A^6]
            if (sub == 0) {
                A.rho[i] = rc;
                A.Fe[i] = F;
                if (OBS) {
                    A.dF2[i] = make_double2(dF, d2F);
                    A.dF2f[i] = make_float2(static_cast<float>(dF / (a3 * kEv)),
                                            static_cast<float>(d2F / (a3 * a3 * kEv)));
                } else {
                    A.dF2[i].x = dF;
                    A.dF2f[i].x = static_cast<float>(dF / (a3 * kEv));
                }
            }
        }
        // the atom's terms of the block sums, equal in its TPA lanes (zero without an atom)
        double v[kP2] = {};
        v[D_FSUM] = F;
        if (OBS) {
            // g in cm^-3 and h in cm^-4, as the cgs F'' expects
            double const ia3 = 1. / a3, iha = 1. / (a3 * kAng);
            double gc[6];
#pragma unroll
            for (int u = 0; u < 6; ++u)
                gc[u] = static_cast<double>(g[u]) * ia3;
            int q = D_CB;
#pragma unroll
            for (int u = 0; u < 6; ++u)
#pragma unroll
                for (int w = u; w < 6; ++w)
                    v[q++ % kP2] = d2F * gc[u] * gc[w];
            double const h0 = hv[0] * iha, h1 = hv[1] * iha, h2 = hv[2] * iha;
            v[D_LAP % kP2] = d2F * (h0 * h0 + h1 * h1 + h2 * h2);
        }
        acc += warp_slots<kP2, TPA>(v);
    }
    // the warps' slots into the block sums; unsampled steps form the embedding energy only
    __shared__ double s_acc[kBlock / 32][kP2];
    int const lane = threadIdx.x & 31;
    if (lane < kP2)
        s_acc[threadIdx.x >> 5][lane_slot<kP2>(lane)] = acc;
    __syncthreads();
    for (int k = threadIdx.x; k < D_NSUM; k += kBlock) {
        double s = 0.;
        if (k < kSlots)
#pragma unroll
            for (int w = 0; w < kBlock / 32; ++w)
                s += s_acc[w][k];
        A.pd[static_cast<size_t>(blockIdx.x) * D_NSUM + k] = s;
    }
}

// Sums over the pairs of one lane's share of an atom row, added into the FP64 block
// accumulators once per row. The diagonal Born stress is summed in FP64 pair by pair and
// the virial is taken as its trace (the sum over pairs of dE/dr r equals that of
// dE/dr x_a^2 / r): the reference checks the virial against the stress trace to 1e-7 and
// the pressure against the stress trace to 1e-5 (md_driver.cpp:422-429, 693-698), and near
// zero pressure, where kinetic and virial parts cancel, that holds only if both come from
// the same FP32 pair terms. The off-diagonal stress, Born tensor and Laplacian terms are
// summed in FP32 along the row (at most ~20 FP32 terms, no error beyond the terms' own)
// and in FP64 across rows and atoms.
template <bool OBS> struct PairSums {
    double sig_d[3] = {0., 0., 0.};
    float sig_o[3] = {0, 0, 0};
    float cb[OBS ? 15 : 1] = {};
    float lap = 0.f;
};

// Per-atom inputs of one row of the force pass.
struct RowIn {
    float4 pi;
    float dFi, d2Fi;
    int ti;
    uint2 slots; // byte b: the pair slot with type b
    float3 L, iL;
};

// The quintic record of phi_s and the derivative records of rho of the pair's types lo <= hi on
// interval k: from the staged shared-memory copy (STAGED and k staged; c0..c5 alone, the
// products formed here) or from the global records. Both give the same FP32 values (a product
// by 2 or 4 is exact), so the pair terms do not depend on where they were read. A pair of one
// type reads its one rho once: dh is left undefined and the caller takes the terms of dl.
//
// phi and rho_lo lie in one 32-byte and one 16-byte record: the L1 data pipe takes 27 and 16
// wavefronts for them, two 32-byte records 54.
template <bool STAGED>
__device__ __forceinline__ void pair_coefs(TablesView const &T, const float *stab, int s,
                                           int lo, int hi, int k, float (&cp)[8],
                                           float (&dl)[8], float (&dh)[8]) {
    if (STAGED) {
        unsigned const q = static_cast<unsigned>(k - T.st_lo);
        if (q < static_cast<unsigned>(T.st_n)) {
            int const n6 = 6 * T.st_n;
            const float *b = stab + 6 * q;
            const float2 *pp = reinterpret_cast<const float2 *>(b + s * n6);
            const float2 *pi = reinterpret_cast<const float2 *>(b + (T.npot + lo) * n6);
            const float2 *pj = reinterpret_cast<const float2 *>(b + (T.npot + hi) * n6);
            float ci[6], cj[6];
#pragma unroll
            for (int u = 0; u < 3; ++u) {
                float2 const a = pp[u], c = pi[u], d = pj[u];
                cp[2 * u] = a.x;
                cp[2 * u + 1] = a.y;
                ci[2 * u] = c.x;
                ci[2 * u + 1] = c.y;
                cj[2 * u] = d.x;
                cj[2 * u + 1] = d.y;
            }
            cp[6] = __fmul_rn(3.f, cp[3]);
            cp[7] = __fmul_rn(5.f, cp[5]);
            derivative_record(ci, dl);
            derivative_record(cj, dh);
            return;
        }
    }
    constexpr int kFf = TabFmt<MDELAST_QUINTIC>::kFf;
    unsigned const q = static_cast<unsigned>(s * T.nri + k);
    float4 const x = __ldg(reinterpret_cast<const float4 *>(T.phq) + q);
    ld256(T.phf + q * kFf, cp);
    ld256_if(lo != hi, T.rdf + static_cast<unsigned>(hi * T.nri + k) * kFf, dh);
    dl[0] = cp[6];
    dl[1] = cp[7];
    dl[2] = x.x;
    dl[3] = x.y;
    dl[4] = x.z;
    dl[5] = __fmul_rn(2.f, x.x);
    dl[6] = __fmul_rn(3.f, x.y);
    dl[7] = __fmul_rn(4.f, x.z);
    cp[6] = x.w;
    cp[7] = __fmul_rn(5.f, cp[5]);
}

// One lane's walk over list slots [s0, s1) of an atom row (slots of the upper half when
// UPPER, else of the lower half, addressed from the end of the row); every pair adds its
// force and half its energy to the atom, and the upper half also adds to the global sums.
// STAGED: quintic tables read from the staged shared-memory copy `stab` where staged. UC: no
// test of a pair's own against the functions' cutoffs or its r_min; dr_min takes the row's smallest
// distance, else -1 when a pair within the cutoff lies below its r_min (potential.hpp:92-104 warns).
template <bool OBS, bool UPPER, int TPA, int IP, bool STAGED, typename IX, bool UC>
__device__ __forceinline__ void force_row_mx(AtomsView const &A, TablesView const &T,
                                             RowIn const &in, PairRow<IX> const &row, int n,
                                             int sub,
                                             double &fx, double &fy, double &fz, double &epot,
                                             PairSums<OBS> &ps, float &dr_min,
                                             const float *stab = nullptr) {
    if (sub >= n)
        return;
    auto slot = [&](int k) { return UPPER ? k : A.pmaxn - 1 - k; };
    // the row's entries are read once per pass: streaming loads (evict first), so that
    // they do not push the table and the partner records out of the L1 (measured: step
    // 1.025 -> 0.987 ms at 16 x 13,500 atoms)
    int jn = row.at(slot(sub));
    float4 pn = A.posf[jn];
    float2 fn = A.dF2f[jn];
    jn = row.at(slot(min(sub + TPA, n - 1)));
    // The body has no branch: a pair beyond the cutoff is evaluated and its terms are
    // replaced by zeros (the sums then gain +0 or -0, which changes no sum), the second rho of
    // a two-type pair is a predicated load, and the next partner is always prefetched (the
    // last one again at the end of the row). Not unrolled: one body fills the 128 registers of
    // 4 blocks per SM, two spill (0.346 instead of 0.312 ms at 16 x 13,500 atoms).
#pragma unroll 1
    for (int kk = sub; kk < n; kk += TPA) {
        float4 const pj = pn;
        float2 const dFj2 = fn;
        pn = A.posf[jn];
        fn = A.dF2f[jn];
        jn = row.at(slot(min(kk + 2 * TPA, n - 1)));
        float dx, dy, dz;
        float const r2 = min_image_f(in.pi, pj, in.L, in.iL, dx, dy, dz);
        bool const in_cut = !(r2 > T.fr_cut_sq);
        float const idr = rsqrtf(r2);
        float const dr = __fmul_rn(r2, idr);
        int const ti = in.ti, tj = __float_as_int(pj.w);
        int const s = __byte_perm(in.slots.x, in.slots.y, tj) & 0xff;
        if (UC)
            dr_min = fminf(dr_min, dr);
        else if (in_cut && dr < T.fpot_rmin[s])
            dr_min = -1.f;
        float t;
        int const k = tab_locate_f(dr, T.finv_hr, T.nri, t);
        float V = 0.f, dV = 0.f, d2V = 0.f;
        float drho_i = 0.f, drho_j = 0.f, d2rho_i = 0.f, d2rho_j = 0.f;
        bool const eam_i = UC || (T.has_eam && !(dr > T.feam_rcut[ti]));
        bool const eam_j = UC || (T.has_eam && !(dr > T.feam_rcut[tj]));
        if constexpr (IP == MDELAST_QUINTIC) {
            // the three functions' coefficients first (independent loads), then the math
            float cp[8], dl[8], dh[8];
            pair_coefs<STAGED>(T, stab, s, min(ti, tj), max(ti, tj), k, cp, dl, dh);
            if (UC || !(dr > T.fpot_rcut[s])) {
                V = tabf_v(cp, t);
                dV = tabf_d1(cp, t, T.finv_hr);
                if (OBS)
                    d2V = tabf_d2(cp, t, T.finv_hr2);
            }
            // rho' and rho'' of the types lo and hi, then of i and j
            float const l1 = tabd_d1(dl, t, T.finv_hr), h1 = tabd_d1(dh, t, T.finv_hr);
            drho_i = ti <= tj ? l1 : h1;
            drho_j = ti < tj ? h1 : l1;
            if (OBS) {
                float const l2 = tabd_d2(dl, t, T.finv_hr2), h2 = tabd_d2(dh, t, T.finv_hr2);
                d2rho_i = ti <= tj ? l2 : h2;
                d2rho_j = ti < tj ? h2 : l2;
            }
            if (!eam_i)
                drho_i = d2rho_i = 0.f;
            if (!eam_j)
                drho_j = d2rho_j = 0.f;
        } else {
            constexpr int kFf = TabFmt<IP>::kFf;
            if (UC || !(dr > T.fpot_rcut[s]))
                tabf_eval<IP, true, true, OBS>(T.phf + static_cast<unsigned>(s * T.nri + k) * kFf,
                                               t, T.finv_hr, T.finv_hr2, V, dV, d2V);
            float unused = 0.f;
            if (eam_i)
                tabf_eval<IP, false, true, OBS>(
                    T.rrf + static_cast<unsigned>(ti * T.nri + k) * kFf, t, T.finv_hr,
                    T.finv_hr2, unused, drho_i, d2rho_i);
            if (eam_j)
                tabf_eval<IP, false, true, OBS>(
                    T.rrf + static_cast<unsigned>(tj * T.nri + k) * kFf, t, T.finv_hr,
                    T.finv_hr2, unused, drho_j, d2rho_j);
        }
        float dedr = dV, X = 0.f, lap = 0.f;
        if (OBS) {
            X = d2V - dV * idr;
            lap = 2.f * (d2V + 2.f * dV * idr);
        }
        if (UC || T.has_eam) {
            float const dFj = dFj2.x, dFi = in.dFi;
            // the two cross terms rounded separately and added commutatively: the pair
            // force is the same, bit for bit, seen from either atom
            dedr = __fadd_rn(dedr, __fadd_rn(__fmul_rn(dFi, drho_j), __fmul_rn(dFj, drho_i)));
            if (OBS && UPPER) {
                float const d2Fj = dFj2.y, d2Fi = in.d2Fi;
                lap += 2.f * (dFj * (d2rho_i + 2.f * drho_i * idr) +
                              dFi * (d2rho_j + 2.f * drho_j * idr));
                lap += d2Fi * (drho_j * drho_j) + d2Fj * (drho_i * drho_i);
                X += dFi * (d2rho_j - drho_j * idr) + dFj * (d2rho_i - drho_i * idr);
            }
        }
        if (!in_cut) {
            dedr = 0.f;
            V = 0.f;
            X = 0.f;
            lap = 0.f;
        }
        float const sc = __fmul_rn(-dedr, idr);
        fx += static_cast<double>(__fmul_rn(sc, dx));
        fy += static_cast<double>(__fmul_rn(sc, dy));
        fz += static_cast<double>(__fmul_rn(sc, dz));
        epot += static_cast<double>(V); // halved at the end of the row
        if (UPPER) {
            float const xx = dx * dx, yy = dy * dy, zz = dz * dz;
            float const yz = dy * dz, xz = dx * dz, xy = dx * dy;
            ps.sig_d[0] -= static_cast<double>(sc * xx); // sc = -dE/dr / r
            ps.sig_d[1] -= static_cast<double>(sc * yy);
            ps.sig_d[2] -= static_cast<double>(sc * zz);
            ps.sig_o[0] -= sc * yz;
            ps.sig_o[1] -= sc * xz;
            ps.sig_o[2] -= sc * xy;
            if (OBS) {
                X *= idr * idr;
                float const Xxx = X * xx, Xyy = X * yy, Xzz = X * zz;
                ps.cb[0] += Xxx * xx;
                ps.cb[1] += Xyy * yy;
                ps.cb[2] += Xzz * zz;
                ps.cb[3] += Xxx * xy;
                ps.cb[4] += Xxx * xz;
                ps.cb[5] += Xyy * xy;
                ps.cb[6] += Xyy * yz;
                ps.cb[7] += Xzz * xz;
                ps.cb[8] += Xzz * yz;
                ps.cb[9] += Xxx * yy;
                ps.cb[10] += Xxx * zz;
                ps.cb[11] += Xyy * zz;
                ps.cb[12] += Xxx * yz;
                ps.cb[13] += Xyy * xz;
                ps.cb[14] += Xzz * xy;
                ps.lap += lap;
            }
        }
    }
}

// Force pass of md_driver.cpp:300-430 (with the closing kick) in mixed precision; see
// k_force for the roles of the terms. Each atom row is walked in two loops, its upper
// half (which also feeds the global sums) and its lower half, so the lanes of a warp do not
// diverge on the global-sum work. The row's 22 pair sums and, after the kick, its 12 sums
// over atoms go through warp_slots (31 and, at 4 lanes per atom, 4 exchanges) into two FP64
// registers per lane; the virial is the trace of the Born stress.
//
// What bounds it: scattered gathers, by their wavefronts (67 per 32 visits, 54 % of the L1 data
// pipe's rate) and their latency at 4 blocks of 4 warps per SM, with instruction issue (47 %) behind. At 16 x 13,500 atoms and 4 lanes per
// atom: 0.416 ms when the sums' shuffles and shared accumulators were 19 % of the data pipe's
// work and the third table function of one-type pairs another 20 %, 0.362 ms without them, 0.345 with
// even row halves, 0.314 with the products of the coefficients in the table records, the r_min test
// once per row, pair slots from a byte table and no unrolling, 0.300 with 48 instead of 64 bytes of
// tables for a one-type pair, 0.296 without the second walk that r_min could ask for.
//
// STAGED: the block first copies the staged quintic tables (T.stf, T.st_bytes, about 180 KB
// for a two-element alloy) into dynamic shared memory and reads every staged interval from
// there, so table lookups no longer compete with the partner gathers for the L1 and never
// miss to the L2. One such block fills an SM's shared memory, so it is NB = kBlockStaged
// threads wide. Per-atom results equal the unstaged kernel's bit for bit; the global sums
// differ only in the grouping of their FP64 partial sums.
constexpr int kBlockStaged = kStagedBlock;

template <bool OBS, bool KICK, int TPA, int IP, bool STAGED, typename IX,
          int NB = STAGED ? kBlockStaged : kBlock>
__global__ void __launch_bounds__(NB, STAGED ? 1 : 4) k_force_mx(AtomsView A, TablesView T) {
    chain_begin();
    if (halted(A)) // a list build ran out of capacity: nothing until the host regrows
        return;
    extern __shared__ float4 s_stage[];
    int const tid = threadIdx.x;
    if (STAGED) {
        const float4 *src = reinterpret_cast<const float4 *>(T.stf);
        int const n16 = T.st_bytes / 16;
        for (int k = tid; k < n16; k += NB)
            s_stage[k] = __ldg(src + k);
        __syncthreads();
    }
    const float *stab = reinterpret_cast<const float *>(s_stage);
    int const r = A.fblk_rep[blockIdx.x];
    Replica const *R = A.rep + r;
    int const lb = blockIdx.x - R->fblk_begin, nb = R->fblk_n;
    int const apb = NB / TPA, sub = tid % TPA;
    int const n_slots = R->n_blocks * kBlock;
    constexpr int kPair = OBS ? F_F2 - F_SIGMA : F_CB - F_SIGMA, kP2 = slots_pow2(kPair);
    constexpr int kKick = F_NSUM - F_F2, kK2 = slots_pow2(kKick);
    double acc_p = 0., acc_k = 0.; // the block sums of this lane's slots
    RowIn in;
    box_f(R, in.L, in.iL);
    for (int a0 = lb * apb; a0 < n_slots; a0 += nb * apb) {
        int const a = a0 + tid / TPA;
        int const i = R->atom_begin + a;
        bool const valid = a < R->n_atoms;
        double fx = 0., fy = 0., fz = 0., epot = 0.;
        double v[kP2] = {}; // this lane's pair sums: Born stress, tensor, Laplacian
        in.ti = 0;
        if (valid) {
            in.pi = A.posf[i];
            in.ti = __float_as_int(in.pi.w);
            in.slots = T.slots[in.ti];
            float2 const dFi2 = T.has_eam ? A.dF2f[i] : make_float2(0.f, 0.f);
            in.dFi = dFi2.x;
            in.d2Fi = OBS ? dFi2.y : 0.f;
            int const nu = A.pn_up[i], nd = A.pn_dn[i];
            PairRow<IX> const row = pair_row<IX>(A, i, R->atom_begin);
            float dr_min = 3.4e38f; // of this lane's pairs
            PairSums<OBS> ps;
            // one cutoff and one r_min (every setfl potential): no tests per function and pair
            // (16 x 13,500 atoms: 0.294 ms; with them, for an r_min of its own per pair type,
            // 0.311; a second walk over the rows with a distance below the largest, 0.472)
            bool const uc = T.fuc && T.frmin >= 0.f;
            if (uc) {
                force_row_mx<OBS, true, TPA, IP, STAGED, IX, true>(
                    A, T, in, row, nu, sub, fx, fy, fz, epot, ps, dr_min, stab);
                force_row_mx<OBS, false, TPA, IP, STAGED, IX, true>(
                    A, T, in, row, nd, sub, fx, fy, fz, epot, ps, dr_min, stab);
            } else {
                force_row_mx<OBS, true, TPA, IP, STAGED, IX, false>(
                    A, T, in, row, nu, sub, fx, fy, fz, epot, ps, dr_min, stab);
                force_row_mx<OBS, false, TPA, IP, STAGED, IX, false>(
                    A, T, in, row, nd, sub, fx, fy, fz, epot, ps, dr_min, stab);
            }
            epot *= 0.5;
            if (dr_min < (uc ? T.frmin : 0.f))
                status_or(A.rep + r, MDELAST_WARN_RMIN);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                v[k] = ps.sig_d[k];
                v[3 + k] = static_cast<double>(ps.sig_o[k]);
            }
            if (OBS) {
#pragma unroll
                for (int k = 0; k < 15; ++k)
                    v[(F_CB - F_SIGMA + k) % kP2] = static_cast<double>(ps.cb[k]);
                v[(F_LAP - F_SIGMA) % kP2] = static_cast<double>(ps.lap);
            }
        }
        acc_p += warp_slots<kP2, 1>(v);
        fx = group_sum<TPA>(fx);
        fy = group_sum<TPA>(fy);
        fz = group_sum<TPA>(fz);
        epot = group_sum<TPA>(epot);
        double vx = 0., vy = 0., vz = 0., m = 0.;
        double w[kK2] = {}; // the atom's terms of the sums over atoms, equal in its lanes
        if (valid) { // every lane of the atom, stored by the first
            double const kf = kEv / kAng; // eV/A -> dyn
            fx *= kf;
            fy *= kf;
            fz *= kf;
            epot *= kEv;
            if (T.has_eam)
                epot += A.Fe[i];
            size_t const np = A.n_pad;
            m = T.mass[in.ti];
            vx = A.vel[i];
            vy = A.vel[np + i];
            vz = A.vel[2 * np + i];
            if (KICK) {
                double const e = R->e_kick, cdt = R->cdt_kick;
                vx = vx * e + cdt * fx / m;
                vy = vy * e + cdt * fy / m;
                vz = vz * e + cdt * fz / m;
            }
        }
        __syncwarp(); // the atom's lanes have read its velocity
        if (valid && sub == 0) {
            size_t const np = A.n_pad;
            A.frc[i] = fx;
            A.frc[np + i] = fy;
            A.frc[np + i + np] = fz;
            A.epot[i] = epot;
            if (KICK) {
                A.vel[i] = vx;
                A.vel[np + i] = vy;
                A.vel[2 * np + i] = vz;
            }
        }
        if (valid) {
            w[F_F2 - F_F2] = fx * fx + fy * fy + fz * fz;
            w[F_EKIN - F_F2] = 0.5 * m * (vx * vx + vy * vy + vz * vz);
            w[F_MVV + 0 - F_F2] = m * vx * vx;
            w[F_MVV + 1 - F_F2] = m * vy * vy;
            w[F_MVV + 2 - F_F2] = m * vz * vz;
            w[F_MVV + 3 - F_F2] = m * vy * vz;
            w[F_MVV + 4 - F_F2] = m * vx * vz;
            w[F_MVV + 5 - F_F2] = m * vx * vy;
            w[F_MV + 0 - F_F2] = vx * m;
            w[F_MV + 1 - F_F2] = vy * m;
            w[F_MV + 2 - F_F2] = vz * m;
            w[F_EPOT - F_F2] = epot;
        }
        acc_k += warp_slots<kK2, TPA>(w);
    }
    // the warps' slots into the block sums; pair sums from eV (and eV/A^2 for the
    // Laplacian) to cgs, the virial as the trace of the Born stress
    __shared__ double s_acc[NB / 32][F_NSUM];
    int const lane = tid & 31, warp = tid >> 5;
    if (lane < kP2 && lane_slot<kP2>(lane) < kPair)
        s_acc[warp][F_SIGMA + lane_slot<kP2>(lane)] = acc_p;
    if (lane < kK2 && lane_slot<kK2>(lane) < kKick)
        s_acc[warp][F_F2 + lane_slot<kK2>(lane)] = acc_k;
    __syncthreads();
    auto block_sum = [&](int k) {
        double s = 0.;
#pragma unroll
        for (int q = 0; q < NB / 32; ++q)
            s += s_acc[q][k];
        return s;
    };
    for (int k = tid; k < F_NSUM; k += NB) {
        double s = 0.;
        if (k == F_VIRIAL)
            s = ((block_sum(F_SIGMA) + block_sum(F_SIGMA + 1)) + block_sum(F_SIGMA + 2)) * kEv;
        else if (k >= F_F2)
            s = block_sum(k);
        else if (k - F_SIGMA < kPair)
            s = block_sum(k) * (k == F_LAP ? kEv / (kAng * kAng) : kEv);
        A.pf[static_cast<size_t>(blockIdx.x) * F_NSUM + k] = s;
    }
}

namespace {
template <bool OBS, int IP, typename IX>
void density_mx_tpa_ix(int tpa, int grid, cudaStream_t s, AtomsView const &A,
                       TablesView const &T) {
    switch (tpa) {
    case 1: launch_pass(tpa, k_density_mx<OBS, 1, IP, IX>, grid, kBlock, 0, s, A, T); break;
    case 4: launch_pass(tpa, k_density_mx<OBS, 4, IP, IX>, grid, kBlock, 0, s, A, T); break;
    case 8: launch_pass(tpa, k_density_mx<OBS, 8, IP, IX>, grid, kBlock, 0, s, A, T); break;
    case 16: launch_pass(tpa, k_density_mx<OBS, 16, IP, IX>, grid, kBlock, 0, s, A, T); break;
    default: launch_pass(tpa, k_density_mx<OBS, 32, IP, IX>, grid, kBlock, 0, s, A, T); break;
    }
}
template <bool OBS, int IP>
void density_mx_tpa(int tpa, int grid, cudaStream_t s, AtomsView const &A, TablesView const &T) {
    if (A.pnbr16)
        density_mx_tpa_ix<OBS, IP, uint16_t>(tpa, grid, s, A, T);
    else
        density_mx_tpa_ix<OBS, IP, int>(tpa, grid, s, A, T);
}
template <bool OBS, bool KICK, int IP, typename IX>
void force_mx_tpa_ix(int tpa, int grid, cudaStream_t s, AtomsView const &A,
                     TablesView const &T) {
    switch (tpa) {
    case 1: launch_pass(tpa, k_force_mx<OBS, KICK, 1, IP, false, IX>, grid, kBlock, 0, s, A, T); break;
    case 4: launch_pass(tpa, k_force_mx<OBS, KICK, 4, IP, false, IX>, grid, kBlock, 0, s, A, T); break;
    case 8: launch_pass(tpa, k_force_mx<OBS, KICK, 8, IP, false, IX>, grid, kBlock, 0, s, A, T); break;
    case 16: launch_pass(tpa, k_force_mx<OBS, KICK, 16, IP, false, IX>, grid, kBlock, 0, s, A, T); break;
    default: launch_pass(tpa, k_force_mx<OBS, KICK, 32, IP, false, IX>, grid, kBlock, 0, s, A, T); break;
    }
}
template <bool OBS, bool KICK, int IP>
void force_mx_tpa(int tpa, int grid, cudaStream_t s, AtomsView const &A, TablesView const &T) {
    if (A.pnbr16)
        force_mx_tpa_ix<OBS, KICK, IP, uint16_t>(tpa, grid, s, A, T);
    else
        force_mx_tpa_ix<OBS, KICK, IP, int>(tpa, grid, s, A, T);
}
// the staged kernels: lanes per atom 4, 8, 16 or 32
template <bool OBS, bool KICK, typename IX>
void force_mx_staged_ix(int tpa, int grid, cudaStream_t s, AtomsView const &A,
                        TablesView const &T) {
    size_t const smem = static_cast<size_t>(T.st_bytes);
    constexpr int Q = MDELAST_QUINTIC;
    switch (tpa) {
    case 4: launch_pass(tpa, k_force_mx<OBS, KICK, 4, Q, true, IX>, grid, kBlockStaged, smem, s, A, T); break;
    case 8: launch_pass(tpa, k_force_mx<OBS, KICK, 8, Q, true, IX>, grid, kBlockStaged, smem, s, A, T); break;
    case 16: launch_pass(tpa, k_force_mx<OBS, KICK, 16, Q, true, IX>, grid, kBlockStaged, smem, s, A, T); break;
    default: launch_pass(tpa, k_force_mx<OBS, KICK, 32, Q, true, IX>, grid, kBlockStaged, smem, s, A, T); break;
    }
}
template <bool OBS, bool KICK>
void force_mx_staged_tpa(int tpa, int grid, cudaStream_t s, AtomsView const &A,
                         TablesView const &T) {
    if (A.pnbr16)
        force_mx_staged_ix<OBS, KICK, uint16_t>(tpa, grid, s, A, T);
    else
        force_mx_staged_ix<OBS, KICK, int>(tpa, grid, s, A, T);
}
template <bool OBS, bool KICK, typename IX> cudaError_t staged_attr_ix(int bytes) {
    constexpr int Q = MDELAST_QUINTIC;
    cudaFuncAttribute const a = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaError_t e = cudaFuncSetAttribute(k_force_mx<OBS, KICK, 4, Q, true, IX>, a, bytes);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_force_mx<OBS, KICK, 8, Q, true, IX>, a, bytes);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_force_mx<OBS, KICK, 16, Q, true, IX>, a, bytes);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_force_mx<OBS, KICK, 32, Q, true, IX>, a, bytes);
    return e;
}
template <bool OBS, bool KICK> cudaError_t staged_attr(int bytes) {
    cudaError_t e = staged_attr_ix<OBS, KICK, int>(bytes);
    if (e == cudaSuccess)
        e = staged_attr_ix<OBS, KICK, uint16_t>(bytes);
    return e;
}
template <int IP>
void density_mx_ip(bool obs, int tpa, int grid, cudaStream_t s, AtomsView const &A,
                   TablesView const &T) {
    if (obs)
        density_mx_tpa<true, IP>(tpa, grid, s, A, T);
    else
        density_mx_tpa<false, IP>(tpa, grid, s, A, T);
}
template <int IP>
void force_mx_ip(bool obs, bool kick, int tpa, int grid, cudaStream_t s, AtomsView const &A,
                 TablesView const &T) {
    if (obs && kick)
        force_mx_tpa<true, true, IP>(tpa, grid, s, A, T);
    else if (obs)
        force_mx_tpa<true, false, IP>(tpa, grid, s, A, T);
    else if (kick)
        force_mx_tpa<false, true, IP>(tpa, grid, s, A, T);
    else
        force_mx_tpa<false, false, IP>(tpa, grid, s, A, T);
}
} // namespace

void launch_density_mx(bool obs, int tpa, int grid, cudaStream_t s, AtomsView const &A,
                       TablesView const &T) {
    if (T.interp == MDELAST_BSPLINE)
        density_mx_ip<MDELAST_BSPLINE>(obs, tpa, grid, s, A, T);
    else
        density_mx_ip<MDELAST_QUINTIC>(obs, tpa, grid, s, A, T);
}

void launch_force_mx(bool obs, bool kick, int tpa, int grid, cudaStream_t s, AtomsView const &A,
                     TablesView const &T) {
    if (T.interp == MDELAST_BSPLINE)
        force_mx_ip<MDELAST_BSPLINE>(obs, kick, tpa, grid, s, A, T);
    else
        force_mx_ip<MDELAST_QUINTIC>(obs, kick, tpa, grid, s, A, T);
}

void launch_force_mx_staged(bool obs, bool kick, int tpa, int grid, cudaStream_t s,
                            AtomsView const &A, TablesView const &T) {
    if (obs && kick)
        force_mx_staged_tpa<true, true>(tpa, grid, s, A, T);
    else if (obs)
        force_mx_staged_tpa<true, false>(tpa, grid, s, A, T);
    else if (kick)
        force_mx_staged_tpa<false, true>(tpa, grid, s, A, T);
    else
        force_mx_staged_tpa<false, false>(tpa, grid, s, A, T);
}

cudaError_t prepare_force_mx_staged(int smem_bytes) {
    cudaError_t e = staged_attr<true, true>(smem_bytes);
    if (e == cudaSuccess)
        e = staged_attr<true, false>(smem_bytes);
    if (e == cudaSuccess)
        e = staged_attr<false, true>(smem_bytes);
    if (e == cudaSuccess)
        e = staged_attr<false, false>(smem_bytes);
    return e;
}

} // namespace mdelast
