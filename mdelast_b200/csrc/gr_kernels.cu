// Pair correlation g(r) of one replica (md_driver.cpp:732-862): every pair i < j with
// min-image distance dr < rmaxg adds one to bin floor(dr / drg) of the total histogram
// and, by type pair, of the partial one; then the reference's normalisations.
//
// Counting is exact: dr comes from the same FP64 operations as the reference's (the
// min-image arithmetic the neighbour list uses, a correctly rounded sqrt and divide), so
// every pair lands in the reference's bin; integer counters make the sum order-free; and
// the normalisation repeats the reference's operation order without contraction, so g(r)
// equals the reference's to the last bit.
//
// Two kernels: k_gr_count with an FP32 estimate, described here, and k_gr_count_far without, for
// what gr_enqueue's rule leaves to it.
//
// Work split: units of one pair of 128-atom tiles (I <= J) of the replica, dealt to as many
// blocks as fit the SMs; the J tile is staged in shared memory and each thread scans half of it for
// its own atom of tile I. A block keeps its histogram in shared memory over all its units and
// flushes it once, when it fits, else counts go straight to the global counters. O(N^2 / 2) pair
// tests: about 91 M for 13,500 atoms.
//
// Each pair's bin is first estimated in FP32, from positions in units of the bin width, with a
// margin that covers the estimate's error (gr_margin); only pairs within the margin of a bin edge
// or of rmaxg (about 1 % at 13,500 atoms) are queued and take the reference's FP64 operations.
// 13,500 atoms, 3,750 bins, two types, total and partial, with the readback: 0.81 -> 0.30 ms (this
// kernel 0.25). Before, every pair took the FP64 min image, square root and division, and a block
// per unit flushed 8,500 counts spread over 15,000 bins, as many global atomics as there are
// pairs. Bound by instruction issue (75 %, 65 instructions per pair test).
#include "gr_kernels.cuh"

#include <algorithm>

#include "device.cuh"

namespace mdelast {

namespace {

constexpr int kGrTile = static_cast<int>(kGrTileAtoms);
constexpr size_t kGrSharedMax = 96 * 1024;

constexpr int kGrThreads = 2 * kGrTile;
constexpr int kGrQueue = 1024;                  // pairs of a unit that wait for the FP64 test
constexpr long kGrFlushUnits = 100000;          // 32-bit counts: flushed before 2^32 pairs
constexpr float kGrMaxMargin = 0.05f;           // beyond it k_gr_count_far counts
// A total histogram beyond shared memory takes k_gr_count_far above this number of units: below, the
// estimate's shorter chain counts, above, its share of the SMs' threads (38,000 bins, far / estimate: 2,048
// atoms 0.175 / 0.163 ms, 4,000 0.184 / 0.194, 42,592 4.21 / 4.91).
constexpr long kGrFarUnits = 148 * 2;
// Partial histograms are kept per block up to kGrSharedFew bytes, beyond that (two blocks or three per
// SM) where at least kGrFew of all pairs lie within rmaxg and would be atomics elsewhere (42,592 atoms, three
// of 8,000 bins: to 8 A 2.17 ms in shared memory, 1.73 not; to half the box 2.99 and above 4).
constexpr size_t kGrSharedFew = 48 * 1024;
constexpr double kGrFew = 0.05;
static_assert(kGrTile == 128, "a queue entry holds two 7-bit tile offsets");

// Bound on |estimate - dr / drg| in bins, for box edges of at most H bins and distances of at most
// u bins. Per coordinate: two positions rounded to FP32 (2^-25 H each), their difference (2^-24 H),
// the box edge (2^-24 H) and the image (2^-25 H), 2^-22 H with room to spare, the same for either
// image near half the box; the three squares, the sum, rsqrt.approx (2^-22.4) and the product
// add less than 2^-21 of the distance.
__host__ __device__ __forceinline__ float gr_margin(float H, float u) {
    return 1.7321f * 2.3842e-7f * H + 4.7684e-7f * u;
}

// the reference's operations: the pair's bin, or -1. From r2_skip on certainly dr >= rmaxg.
__device__ __forceinline__ double gr_r2_skip(GrArgs const &g) {
    return g.rmaxg * g.rmaxg * (1. + 1e-12);
}
__device__ __forceinline__ int gr_bin_exact(GrArgs const &g, double4 ci, double4 cj, double hx,
                                            double hy, double hz, double r2_skip) {
    double px, py, pz;
    double const r2 = min_image_r2(ci, cj, hx, hy, hz, px, py, pz);
    if (r2 >= r2_skip)
        return -1;
    double const dr = __dsqrt_rn(r2);
    if (!(dr < g.rmaxg))
        return -1;
    int const b = static_cast<int>(floor(__ddiv_rn(dr, g.drg)));
    return b < g.n_rg ? b : -1; // unreachable for evenly spaced rg; the reference asserts it
}

// Counters: mode 0 the total histogram; modes 1 and 2 the partial ones, whose sum is the total
// (k_gr_norm). In shared memory they start at row 0, in g.counts the partial ones at row 1.
// SHARED: the block's histogram lies in shared memory.
template <bool SHARED, bool PARTIAL>
__global__ void __launch_bounds__(kGrThreads) k_gr_count(GrArgs g, long units) {
    extern __shared__ unsigned s_hist[];
    __shared__ float4 sj[kGrTile];
    __shared__ unsigned short s_queue[kGrQueue];
    __shared__ int s_n;
    int const rows = PARTIAL ? g.ntypes * (g.ntypes + 1) / 2 : 1, nbins = rows * g.n_rg;
    unsigned long long *const counts = g.counts + (PARTIAL ? g.n_rg : 0);
    if (SHARED)
        for (int k = threadIdx.x; k < nbins; k += kGrThreads)
            s_hist[k] = 0u;
    double const hx = g.rep->h[0], hy = g.rep->h[1], hz = g.rep->h[2], r2_skip = gr_r2_skip(g);
    // positions and box in bins
    double const sx = hx / g.drg, sy = hy / g.drg, sz = hz / g.drg;
    float const Lx = static_cast<float>(sx), Ly = static_cast<float>(sy), Lz = static_cast<float>(sz);
    float const iLx = 1.f / Lx, iLy = 1.f / Ly, iLz = 1.f / Lz;
    float const umax = static_cast<float>(g.rmaxg / g.drg);
    float const margin = gr_margin(fmaxf(Lx, fmaxf(Ly, Lz)), umax);
    // estimates below u_in are within rmaxg, from u_out on outside
    float const u_in = umax - margin, u_out = umax + margin;
    float const f_in = 0.5f - margin; // |fraction - 1/2| below it: away from both bin edges
    auto in_bins = [&](double4 c) {
        return make_float4(static_cast<float>((c.x - nint_ref(c.x)) * sx),
                           static_cast<float>((c.y - nint_ref(c.y)) * sy),
                           static_cast<float>((c.z - nint_ref(c.z)) * sz),
                           __int_as_float(static_cast<int>(c.w)));
    };
    auto count = [&](int b, int ti, int tj) {
        int const at = (PARTIAL ? pair_slot(ti, tj) : 0) * g.n_rg + b;
        if (SHARED)
            atomicAdd(&s_hist[at], 1u);
        else
            atomicAdd(&counts[at], 1ull);
    };
    auto flush = [&]() {
        __syncthreads();
        for (int k = threadIdx.x; k < nbins; k += kGrThreads)
            if (unsigned const c = s_hist[k]) {
                atomicAdd(&counts[k], static_cast<unsigned long long>(c));
                s_hist[k] = 0u;
            }
    };
    int const T = (g.n + kGrTile - 1) / kGrTile;
    int const il = threadIdx.x & (kGrTile - 1), half = threadIdx.x / kGrTile;
    int const warp0 = (threadIdx.x & ~31) & (kGrTile - 1); // the warp's first atom of the tile
    // unit q -> tile pair (I, J), I <= J: rows of the upper triangle of T x T tiles, walked as q grows
    long row0 = 0; // first unit of row I
    int I = 0;
    for (long q = blockIdx.x, done = 1; q < units; q += gridDim.x, ++done) {
        while (q - row0 >= T - I) {
            row0 += T - I;
            ++I;
        }
        int const J = I + static_cast<int>(q - row0), i0 = I * kGrTile, j0 = J * kGrTile;
        int const kmax = min(kGrTile, g.n - j0);
        __syncthreads(); // the previous unit is done with the tile and the queue
        for (int k = threadIdx.x; k < kmax; k += kGrThreads)
            sj[k] = in_bins(g.crd[j0 + k]);
        if (threadIdx.x == 0)
            s_n = 0;
        __syncthreads();
        if (i0 + il < g.n) {
            float4 const pi = in_bins(g.crd[i0 + il]);
            int const ti = __float_as_int(pi.w);
            int const kb = half * (kGrTile / 2), ke = min(kmax, kb + kGrTile / 2);
            // the diagonal tile counts only j > i
            int const kfirst = I == J ? il + 1 : 0;
#pragma unroll 2
            for (int k = I == J ? max(kb, warp0) : kb; k < ke; ++k) {
                float4 const pj = sj[k];
                float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
                dx = fmaf(-Lx, round_small(dx * iLx), dx);
                dy = fmaf(-Ly, round_small(dy * iLy), dy);
                dz = fmaf(-Lz, round_small(dz * iLz), dz);
                float const r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
                float const u = r2 * rsqrtf(fmaxf(r2, 1e-30f));
                // floor(u) as the mantissa of u + 2^23 rounded down (estimates below 2^22)
                float const up = __fadd_rd(u, 8388608.f), f = u - (up - 8388608.f);
                int const b = __float_as_int(up) - 0x4b000000;
                bool const sure = u < u_in && fabsf(f - 0.5f) < f_in;
                if (sure && k >= kfirst && b < g.n_rg)
                    count(b, ti, __float_as_int(pj.w));
                if (sure || k < kfirst || u >= u_out)
                    continue;
                int const at = atomicAdd(&s_n, 1);
                if (at < kGrQueue) {
                    s_queue[at] = static_cast<unsigned short>(il << 7 | k);
                } else {
                    double4 const cj = g.crd[j0 + k];
                    int const b = gr_bin_exact(g, g.crd[i0 + il], cj, hx, hy, hz, r2_skip);
                    if (b >= 0)
                        count(b, ti, static_cast<int>(cj.w));
                }
            }
        }
        __syncthreads();
        for (int e = threadIdx.x; e < min(s_n, kGrQueue); e += kGrThreads) {
            double4 const ci = g.crd[i0 + (s_queue[e] >> 7)], cj = g.crd[j0 + (s_queue[e] & 127)];
            int const b = gr_bin_exact(g, ci, cj, hx, hy, hz, r2_skip);
            if (b >= 0)
                count(b, static_cast<int>(ci.w), static_cast<int>(cj.w));
        }
        if (SHARED && done % kGrFlushUnits == 0)
            flush();
    }
    if (SHARED)
        flush();
}

// Every pair by the reference's operations, straight to the global counters, a block per unit: for
// bins too fine for the estimate, and for a total histogram beyond shared memory, where the atomics
// are the bound and the estimate gains nothing. In k_gr_count, bins too fine queued every pair, those
// beyond rmaxg too: 42,592 atoms, bins of 0.0005 A to 6 A, 4.84 ms, here 1.71; bins of 0.0004 A to half
// the box (100,000), total 5.72 ms, here 3.11.
template <bool PARTIAL>
__global__ void __launch_bounds__(kGrTile) k_gr_count_far(GrArgs g) {
    __shared__ double4 sj[kGrTile];
    int const T = (g.n + kGrTile - 1) / kGrTile;
    long q = blockIdx.x;
    int I = 0;
    for (; q >= T - I; ++I)
        q -= T - I;
    int const j0 = (I + static_cast<int>(q)) * kGrTile, kmax = min(kGrTile, g.n - j0);
    for (int k = threadIdx.x; k < kmax; k += kGrTile)
        sj[k] = g.crd[j0 + k];
    __syncthreads();
    double const hx = g.rep->h[0], hy = g.rep->h[1], hz = g.rep->h[2], r2_skip = gr_r2_skip(g);
    int const i = I * kGrTile + static_cast<int>(threadIdx.x);
    if (i >= g.n)
        return;
    double4 const ci = g.crd[i];
    int const ti = static_cast<int>(ci.w);
    // the diagonal tile counts only j > i
#pragma unroll 4
    for (int k = q == 0 ? static_cast<int>(threadIdx.x) + 1 : 0; k < kmax; ++k) {
        double4 const cj = sj[k];
        int const b = gr_bin_exact(g, ci, cj, hx, hy, hz, r2_skip);
        if (b >= 0)
            atomicAdd(&g.counts[(PARTIAL ? 1 + pair_slot(ti, static_cast<int>(cj.w)) : 0) * g.n_rg + b],
                      1ull);
    }
}

__global__ void k_count_types(GrArgs g) {
    __shared__ int s_t[kMaxTypes]; // one global atomic per block and type
    if (threadIdx.x < kMaxTypes)
        s_t[threadIdx.x] = 0;
    __syncthreads();
    int const i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < g.n)
        atomicAdd(&s_t[static_cast<int>(g.crd[i].w)], 1);
    __syncthreads();
    if (static_cast<int>(threadIdx.x) < g.ntypes && s_t[threadIdx.x])
        atomicAdd(&g.n_per_type[threadIdx.x], s_t[threadIdx.x]);
}

// md_driver.cpp:749-751 (total) and :786-810 (partial), in the reference's operation order
__global__ void k_gr_norm(GrArgs g) {
    int const k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= g.n_rg)
        return;
    double const pi = 3.14159265358979323846;
    // Box::volume of a diagonal box: h00 * (h11 * h22), the other cofactor terms vanish
    double const V = __dmul_rn(g.rep->h[0], __dmul_rn(g.rep->h[1], g.rep->h[2]));
    double const r = g.rg[k];
    if (g.mode == 0 || g.mode == 1) {
        double const nd = static_cast<double>(g.n);
        unsigned long long total = g.mode == 0 ? g.counts[k] : 0ull;
        for (int q = 0; g.mode == 1 && q < g.ntypes * (g.ntypes + 1) / 2; ++q)
            total += g.counts[(1 + q) * g.n_rg + k];
        double const den =
            __dmul_rn(__dmul_rn(__dmul_rn(__dmul_rn(__dmul_rn(2. * pi, nd), nd), r), r), g.drg);
        g.gr[k] = __dmul_rn(static_cast<double>(total), __ddiv_rn(V, den));
    }
    if (g.mode == 1 || g.mode == 2) {
        int s = 0;
        for (int b = 0; b < g.ntypes; ++b)
            for (int a = 0; a <= b; ++a, ++s) {
                double const Na = static_cast<double>(g.n_per_type[a]);
                double const Nb = static_cast<double>(g.n_per_type[b]);
                double pc = 0.;
                if (a == b) {
                    if (Na > 1)
                        pc = __ddiv_rn(__dmul_rn(Na, __dadd_rn(Na, -1.)), 2.);
                } else {
                    pc = __dmul_rn(Na, Nb);
                }
                double v = 0.;
                if (pc > 0.) {
                    double const pref = __ddiv_rn(V, __dmul_rn(__dmul_rn(4. * pi, pc), g.drg));
                    v = __dmul_rn(static_cast<double>(g.counts[(1 + s) * g.n_rg + k]),
                                  __ddiv_rn(pref, __dmul_rn(r, r)));
                }
                g.gr_partial[static_cast<size_t>(s) * g.n_rg + k] = v;
            }
    }
}

} // namespace

cudaError_t gr_enqueue(GrArgs const &g, cudaStream_t s) {
    size_t const nbins = gr_count_slots(g.n_rg, g.ntypes);
    cudaError_t e = cudaMemsetAsync(g.counts, 0, sizeof(unsigned long long) * nbins, s);
    if (e == cudaSuccess)
        e = cudaMemsetAsync(g.n_per_type, 0, sizeof(int) * g.ntypes, s);
    if (e != cudaSuccess)
        return e;
    if (g.n >= 2) {
        long const units = gr_count_blocks(g.n);
        int const rows = g.mode != 0 ? g.ntypes * (g.ntypes + 1) / 2 : 1;
        size_t const hist = sizeof(unsigned) * static_cast<size_t>(rows) * g.n_rg;
        // the part of all pairs that lies within rmaxg
        double const V = g.box[0] * (g.box[1] * g.box[2]);
        double const part = 4.2 * g.rmaxg * g.rmaxg * g.rmaxg / V;
        double const edge = std::max(g.box[0], std::max(g.box[1], g.box[2]));
        bool const estimate = gr_margin(static_cast<float>(edge / g.drg),
                                        static_cast<float>(g.rmaxg / g.drg)) < kGrMaxMargin;
        bool const shared_hist = hist <= kGrSharedMax && (g.mode == 0 || hist <= kGrSharedFew || part > kGrFew);
        if (!estimate || (g.mode == 0 && !shared_hist && units > kGrFarUnits)) {
            auto const far = g.mode == 0 ? k_gr_count_far<false> : k_gr_count_far<true>;
            far<<<static_cast<unsigned>(units), kGrTile, 0, s>>>(g);
        } else {
            size_t const smem = shared_hist ? hist : 0;
            auto const kernel = g.mode != 0 ? (shared_hist ? k_gr_count<true, true> : k_gr_count<false, true>)
                                            : (shared_hist ? k_gr_count<true, false> : k_gr_count<false, false>);
            if (shared_hist)
                e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(kGrSharedMax));
            int per_sm = 1;
            if (e == cudaSuccess)
                e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kGrThreads, smem);
            if (e != cudaSuccess)
                return e;
            long const blocks = std::min(units, 148L * std::max(per_sm, 1));
            kernel<<<static_cast<unsigned>(blocks), kGrThreads, smem, s>>>(g, units);
        }
    }
    if (g.n > 0)
        k_count_types<<<(g.n + 255) / 256, 256, 0, s>>>(g);
    k_gr_norm<<<(g.n_rg + 255) / 256, 256, 0, s>>>(g);
    return cudaGetLastError();
}

} // namespace mdelast
