// Device helpers shared by the FP64 and the mixed-precision pair kernels.
#pragma once

#include "device.cuh"

namespace mdelast {

__device__ __forceinline__ void status_or(Replica *rep, unsigned bits) {
    atomicOr(&rep->obs.status, bits);
}

// a list build ran out of capacity: the rest of the launch's steps are skipped
__device__ __forceinline__ bool halted(AtomsView const &A) { return *A.halt != 0; }
__device__ __forceinline__ void set_halt(AtomsView const &A) { *A.halt = 1; }

// 32 bytes (32-byte aligned) in one 256-bit load through the read-only path.
__device__ __forceinline__ void ld256(const float *p, float (&v)[8]) {
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]),
          "=f"(v[7])
        : "l"(p));
}

// One atom's coordinates and type (32-byte aligned) in one 256-bit load: 27 L1 wavefronts per
// scattered warp instead of 32 for two 128-bit loads (FP64 density + force pass of 54,000 atoms
// 0.240 -> 0.232 ms). Volatile: never before chain_begin().
__device__ __forceinline__ double4 ld_crd(const double4 *p) {
    double4 v;
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
                 : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w)
                 : "l"(p));
    return v;
}

// The same where `on`; elsewhere v is left undefined.
__device__ __forceinline__ void ld256_if(bool on, const float *p, float (&v)[8]) {
    asm("{\n\t"
        ".reg .pred q;\n\t"
        "setp.ne.b32 q, %9, 0;\n\t"
        "@q ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n\t"
        "}"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]),
          "=f"(v[7])
        : "l"(p), "r"(static_cast<int>(on)));
}

// Positions of the mixed passes (AtomsView::posf) from the FP64 scaled coordinates and the box:
// wrapped, in angstrom, the type's bits in .w.
__device__ __forceinline__ float4 position_f(double4 c, Replica const *R) {
    double const u = 1e8; // cm -> angstrom
    return make_float4(static_cast<float>((c.x - nint_ref(c.x)) * R->h[0] * u),
                       static_cast<float>((c.y - nint_ref(c.y)) * R->h[1] * u),
                       static_cast<float>((c.z - nint_ref(c.z)) * R->h[2] * u),
                       __int_as_float(static_cast<int>(c.w)));
}
// minimum image of pi - pj in a box of edges L (positions wrapped into [-L/2, L/2)) and its
// square. Every operation is an odd function: the image seen from j is the negative, bit for bit.
__device__ __forceinline__ float min_image_f(float4 pi, float4 pj, float3 L, float3 iL,
                                             float &dx, float &dy, float &dz) {
    dx = __fsub_rn(pi.x, pj.x);
    dy = __fsub_rn(pi.y, pj.y);
    dz = __fsub_rn(pi.z, pj.z);
    dx = __fmaf_rn(-L.x, round_small(__fmul_rn(dx, iL.x)), dx);
    dy = __fmaf_rn(-L.y, round_small(__fmul_rn(dy, iL.y)), dy);
    dz = __fmaf_rn(-L.z, round_small(__fmul_rn(dz, iL.z)), dz);
    return __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
}

__device__ __forceinline__ void box_f(Replica const *R, float3 &L, float3 &iL) {
    L = make_float3(static_cast<float>(R->h[0] * 1e8), static_cast<float>(R->h[1] * 1e8),
                    static_cast<float>(R->h[2] * 1e8));
    iL = make_float3(__frcp_rn(L.x), __frcp_rn(L.y), __frcp_rn(L.z));
}

// The warp's totals of N per-lane values, one total per lane: at each butterfly level a
// lane keeps half of its values and hands the other half to its partner lane, so N values
// take 31 exchanges instead of the 5 N of N separate warp sums, and the totals end spread over the
// lanes, where a register per lane accumulates them from atom group to atom group. SAME:
// lanes that differ only in the bits below SAME hold equal values that count once (the lanes
// of an atom, after group_sum); those levels only select. Fixed order, so deterministic.
// v holds slots_pow2(N) values, zeros past N; lane l < slots_pow2(N) ends with the total of slot
// lane_slot<slots_pow2(N)>(l).
constexpr __host__ __device__ int slots_pow2(int n) {
    int p = 1;
    while (p < n)
        p <<= 1;
    return p;
}
template <int CUR, int O, int SAME, int P2>
__device__ __forceinline__ void warp_slots_level(double (&v)[P2]) {
    int const lane = threadIdx.x & 31;
    if constexpr (CUR > 1) {
        constexpr int kHalf = CUR / 2;
        bool const up = (lane & O) != 0;
#pragma unroll
        for (int k = 0; k < kHalf; ++k) {
            double const keep = up ? v[kHalf + k] : v[k];
            if constexpr (O < SAME) {
                v[k] = keep;
            } else {
                double const give = up ? v[k] : v[kHalf + k];
                v[k] = keep + __shfl_xor_sync(0xffffffffu, give, O);
            }
        }
    } else if constexpr (O >= SAME) {
        v[0] += __shfl_xor_sync(0xffffffffu, v[0], O);
    }
    if constexpr (O < 16)
        warp_slots_level<(CUR > 1 ? CUR / 2 : 1), 2 * O, SAME>(v);
}
template <int P2, int SAME> __device__ __forceinline__ double warp_slots(double (&v)[P2]) {
    static_assert(P2 <= 32, "one slot per lane");
    warp_slots_level<P2, 1, SAME>(v);
    return v[0];
}
template <int P2> __device__ __forceinline__ int lane_slot(int lane) {
    int s = 0;
#pragma unroll
    for (int o = 1, half = P2 / 2; half > 0; o <<= 1, half >>= 1)
        s += (lane & o) ? half : 0;
    return s;
}

// TPA lanes (a power of two dividing 32) share one atom: lane `sub` takes the atom's list
// entries sub, sub + TPA, ... and the per-atom sums are combined across the lanes with
// shuffles. Every lane must reach the shuffles (padding lanes add zeros).
template <int TPA, typename V> __device__ __forceinline__ V group_sum(V x) {
#pragma unroll
    for (int o = TPA / 2; o > 0; o >>= 1)
        x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// list entry kk of an atom row: the upper half at slots 0.., the lower half at slots maxn-1 down
__device__ __forceinline__ int list_slot(int kk, int nu, int maxn) {
    return kk < nu ? kk : maxn - 1 - (kk - nu);
}

} // namespace mdelast
