// K2+K3+K4: fused three-phonon scattering for one accepted irreducible q-triplet per
// CTA iteration (persistent grid-stride loop over the triplet list).
//
// Reference (src/thermal_conductivity/scattering_threephonon.f90):
//   pretransform_phi3 (:275-317)   ptf(a,b,c) = sum_t mwm_t(i,j,k) exp(-2 pi i (q2.lv2 + q3.lv3))
//   zgeru x2 + dot_product (:93-113)  c0 = sum_abc e1(a) e2(b) e3(c) ptf(a,b,c), e = egv/sqrt(omega)
//   get_dirac (:219-271) and accumulation (:115-135) for Gamma and the Xi row terms.
// The reference recomputes ptf and evp for every b1 of q1 and contracts per (b2,b3)
// (2 n^5 complex MACs per row); here one CTA builds ptf once per q-triplet and contracts
// it with all three eigenvector matrices for all (b1,b2,b3) at once:
//   T1[b1][b][c] = sum_a E1[a][b1] P[a][b][c]
//   T2[b1][b2][c] = sum_b E2[b][b2] T1[b1][b][c]
//   Psi[b1][b2][b3] = sum_c E3[c][b3] T2[b1][b2][c]          (3 n^4 complex MACs)
// The phase factors are exact roots of unity: q = g/N on the mesh and lv are integer
// lattice vectors, so q.lv = sum_d g_d lv_d / N_d and exp(-2 pi i q.lv) is one entry of a
// table of exp(-2 pi i K / L), L = lcm of the mesh dimensions.
//
// With adaptive widths few mode triplets have a Gaussian inside its 8-sigma window (2 % at
// rocksalt 24^3, 3-12 % at 9 to 15 modes), and at two atoms 67 % (12^3) to 76 % (24^3) of the
// q-triplets have none, so the screen comes before the contraction and the contraction is driven by it:
//   1. every mode triplet and each of the four Gaussians of get_dirac is screened in FP32
//      against the window, with a relative margin of 1e-3 and an absolute margin far above
//      FP32 rounding (a Gaussian the screen drops is exactly 0 in the reference); the
//      reference's skip rules are tests of the same loop. A q-triplet without survivors ends
//      here: its terms are exactly 0;
//   2. pretransform and the first stage (n^4 complex MACs), in place;
//   3. the second stage for the (b1, b2) that have a survivor, the third for the survivors
//      alone, a thread each, followed by their weights with the reference's own window test
//      and formulas.
// Each value that is formed is the same sum in the same order as in the full contraction.
// Bound: FP64 runs the FP64 pipe (2 lanes per clock and SM): perovskite 8^3 5.6 -> 3.1 ms,
// L1_2 9^3 (-it 6) 6.4 -> 2.2 ms; mixed precision at n = 6 instruction issue and the latency
// of the phases: rocksalt 24^3 14.6 -> 4.3 ms.
//
// Everything for one triplet lives in shared memory. Precision R is double (FP64 path)
// or float (mixed path: FP32 pretransform and contraction, FP32 delta weights,
// occupations and FP64 accumulation).
#include <cuda_runtime.h>

#include "dev_common.cuh"
#include "k3_parts.cuh"
#include "tdg_internal.cuh"

namespace tdg {

namespace {

constexpr int kPhaseChunk = 512;
// Phase factors held in shared memory at a time: at least kPhaseChunk, more when the survivor
// queue, which takes their place afterwards, is larger anyway (n = 15 in FP32: 1680; in the
// adjoint, where it takes that of two eigenvector matrices as well, 1232).
__host__ __device__ constexpr int phase_chunk(int n, int cs, bool adj) {
    const int room = (4 * n * n * n - (adj ? 2 * cs * n * n : 0)) / cs / 16 * 16;
    return room > kPhaseChunk ? room : kPhaseChunk;
}
// b1 per pass of the second and third stages: all of them where their two n^3 buffers leave
// CTAs enough on an SM, else so many that they do (FP64 at n = 15: one buffer of n^3 and one
// of n^3 / 3, two CTAs instead of one). The adjoint needs both buffers whole.
__host__ __device__ constexpr int b1_pass(int n, int cs, bool adj) {
    return adj || cs == 8 || n < 12 ? n : (n == 15 ? 5 : 6);
}

template <typename R>
__device__ __forceinline__ const R *mwm_ptr(const Fc3Dev &fc);
template <>
__device__ __forceinline__ const double *mwm_ptr<double>(const Fc3Dev &fc) {
    return fc.mwm;
}
template <>
__device__ __forceinline__ const float *mwm_ptr<float>(const Fc3Dev &fc) {
    return fc.mwm32;
}

template <typename C>
__device__ __forceinline__ C twiddle_at(const Fc3Dev &fc, int k);
template <>
__device__ __forceinline__ double2 twiddle_at<double2>(const Fc3Dev &fc, int k) {
    return fc.twiddle[k];
}
template <>
__device__ __forceinline__ float2 twiddle_at<float2>(const Fc3Dev &fc, int k) {
    return fc.twiddle32[k];
}

template <typename C>
__device__ __forceinline__ const C *egvs_ptr(const PhononDev &ph);
template <>
__device__ __forceinline__ const double2 *egvs_ptr<double2>(const PhononDev &ph) {
    return ph.egvs;
}
template <>
__device__ __forceinline__ const float2 *egvs_ptr<float2>(const PhononDev &ph) {
    return ph.egvs32;
}

// The adjoint accumulates d L / d mwm per CTA: FP64 runs in FP64 (in shared memory when the
// n_fc3 * 27 entries fit, else straight into the CTA's FP64 slice in global memory); mixed
// runs in FP32 (flushed every kAdjFlush q-triplets from shared memory) into a slice of
// floats, summed over the slices in FP64 afterwards. GB300's FP64 pipe runs at 1/64 of the
// FP32 rate and every q-triplet adds into all n_fc3 * 27 entries: FP64 additions and
// conversions there were half of the mixed adjoint's FP64 pipe, and 4-byte slices keep the
// per-CTA slices of a large force-constant set (456 x 120 KB at n_fc3 = 1115) in L2 where
// (hi, lo) pairs spilled to DRAM. A slice takes a few hundred q-triplets' terms.
constexpr int kAdjFlush = 64;

// exp(-2 pi i (q2.lv2 + q3.lv3)) of force-constant triplet t as an exact root of unity:
// q = g/N on the mesh and lv integer, so the phase is twiddle[K] with
// K = sum_d ((g2_d lv2_d + g3_d lv3_d) mod N_d) L/N_d mod L, L = lcm(N). Since N_d (L/N_d) = L
// the inner reductions can be dropped: K = (sum_d (g2_d L/N_d) lv2_d + (g3_d L/N_d) lv3_d)
// mod L, the same integer with one division instead of four; u2, u3 hold g_d L/N_d of the
// q-triplet.
template <typename C>
__device__ __forceinline__ C phase3(const Fc3Dev &fc, const MeshDev &m, const int *u2, const int *u3, int t) {
    const int32_t *lv = fc.lv + (size_t)t * 6;
    int S = 0;
#pragma unroll
    for (int d = 0; d < 3; ++d) S += u2[d] * lv[d] + u3[d] * lv[3 + d];
    int K = S % m.L;
    if (K < 0) K += m.L;
    return twiddle_at<C>(fc, K);
}


// Shared-memory layout (bytes) for mode count n and complex size cs.
struct Layout {
    size_t om1, om2, om3, inv1, be2, be3, s1, s2, s3, wrow, w6, r2, f32, bits, E1, E2, E3, ph, Q, pairs, A, B, rowid,
        red, wsum, xb, total;
};
__host__ __device__ inline size_t align16(size_t x) { return (x + 15) & ~size_t(15); }
__host__ __device__ inline Layout make_layout(int n, int cs, bool adj = false) {
    Layout L;
    size_t o = 0;
    const size_t dn = align16(sizeof(double) * n);
    const size_t n2 = (size_t)n * n, n3 = n2 * n;
    L.om1 = o; o += dn;
    L.om2 = o; o += dn;
    L.om3 = o; o += dn;
    L.inv1 = o; o += dn;
    L.be2 = o; o += dn;
    L.be3 = o; o += dn;
    L.s1 = o; o += dn;
    L.s2 = o; o += dn;
    L.s3 = o; o += dn;
    L.wrow = o; o += dn;
    L.r2 = o; o += align16(sizeof(double) * n2);
    L.f32 = o; o += align16(sizeof(float) * n * 12);           // om1..3, s1..3, om lo parts, be2, be3, wrow in FP32
    L.bits = o; o += align16(sizeof(uint32_t) * 2 * n2);       // row/col bits of the non-zero F
    const size_t ez = align16(cs * n2);
    const size_t eph = align16((size_t)cs * phase_chunk(n, cs, adj)), qsz = align16(sizeof(uint32_t) * n3);
    if (adj) {
        // the queue, filled after the second stage, takes the place of E1, E2 and the phases
        // (the back-contraction loads the matrices again): at n = 18 in FP64 the two n^3
        // buffers leave no more room
        L.E3 = o; o += ez;
        L.Q = L.E1 = o;
        L.E2 = o + ez;
        L.ph = o + 2 * ez;
        o += 2 * ez + eph > qsz ? 2 * ez + eph : qsz;
    } else {
        // the phases are dead after the pretransform: the survivor queue takes their place
        L.E1 = o; o += ez;
        L.E2 = o; o += ez;
        L.E3 = o; o += ez;
        L.Q = L.ph = o; o += eph > qsz ? eph : qsz;
        L.w6 = o; o += align16(sizeof(double) * 3 * n2);       // -it 6: widths of the mode pairs
    }
    L.pairs = o; o += align16(sizeof(uint16_t) * n2);          // the (b1, b2) with survivors
    // A: n^3 complex values, then (dense F, a slab of n^2 complex per b1) n^3 doubles; B: the
    // second stage of the b1 of a pass (the adjoint: of all), then 3 n^2 doubles
    L.A = o; o += align16(cs * n3);
    if (adj) L.w6 = L.A;                                       // for the screen only
    const size_t bsz = (size_t)cs * b1_pass(n, cs, adj) * n2, dsz = sizeof(double) * 3 * n2;
    L.B = o; o += align16(bsz > dsz ? bsz : dsz);
    L.rowid = o; o += align16(sizeof(int) * n);
    L.red = o; o += align16(sizeof(int2) * kMaxRed);
    L.wsum = o; o += align16(sizeof(int) * 48);                // block scan [33], pass starts in queue and pairs
    // the adjoint does not mark rows and columns: its xi_bar sums over b2 (n^2 doubles)
    L.xb = L.bits;
    L.total = o;
    return L;
}

__host__ __device__ constexpr int threads_for(int n) { return ((n * n + 31) / 32) * 32; }
// Resident CTAs per SM the register budget is sized for; FP64 buffers at n >= 12 already
// limit residency through shared memory. At n = 6 the FP32 forward pass runs faster with 16
// CTAs of 64 threads at 64 registers (a few spills) than with 12; the FP64 pass and the
// adjoint, with their larger live state, keep 12.
__host__ __device__ constexpr int min_blocks_for(int n, bool dbl, bool adj) {
    return n <= 3 ? 16
                  : (n <= 6 ? (adj || dbl ? 12 : 16)
                            : (n <= 9 ? 6 : (dbl ? (adj ? (n <= 12 ? 2 : 1) : (n <= 12 ? 3 : (n <= 15 ? 2 : 1)))
                                                 : (n <= 15 ? 3 : 2))));
}

// ADJ = false: Gamma and the Xi row terms. ADJ = true: the adjoint pass, which recomputes
// the same Psi and delta weights and accumulates d L / d mwm for the row cotangents a.lam.
template <int N, typename R, bool ADJ>
__global__ void __launch_bounds__(threads_for(N), min_blocks_for(N, sizeof(R) == 8, ADJ)) k_threephonon(ThreePhArgs a) {
    using C = typename CT<R>::C;
    constexpr int N2 = N * N, N3 = N2 * N;
    constexpr int NA = N / 3;
    constexpr int NB1 = b1_pass(N, sizeof(C), ADJ), PASSES = N / NB1;
    static_assert(PASSES * NB1 == N, "passes of equal size");
    constexpr int FS = N2 * (int)(sizeof(C) / sizeof(double));  // doubles per b1 slab of A
    extern __shared__ __align__(16) unsigned char smem[];
    const Layout L = make_layout(N, sizeof(C), ADJ);
    float *f32 = (float *)(smem + L.f32);
    C *E1 = (C *)(smem + L.E1);
    C *E2 = (C *)(smem + L.E2);
    C *E3 = (C *)(smem + L.E3);
    C *ph = (C *)(smem + L.ph);
    uint16_t *pairs = (uint16_t *)(smem + L.pairs);
    C *A = (C *)(smem + L.A);
    C *B = (C *)(smem + L.B);
    double *F = (double *)A;
    double *W6 = (double *)(smem + L.w6);
    K3Smem S;
    S.om1 = (double *)(smem + L.om1); S.om2 = (double *)(smem + L.om2); S.om3 = (double *)(smem + L.om3);
    S.inv1 = (double *)(smem + L.inv1); S.be2 = (double *)(smem + L.be2); S.be3 = (double *)(smem + L.be3);
    S.s1 = (double *)(smem + L.s1); S.s2 = (double *)(smem + L.s2); S.s3 = (double *)(smem + L.s3);
    S.wrow = (double *)(smem + L.wrow);
    S.R2 = (double *)(smem + L.r2);
    S.R3 = (double *)B; S.R2s = S.R3 + N2; S.R3s = S.R2s + N2;  // B is free when the sums start
    S.F = F;
    S.fo1 = f32; S.fo2 = f32 + N; S.fo3 = f32 + 2 * N; S.fs1 = f32 + 3 * N; S.fs2 = f32 + 4 * N; S.fs3 = f32 + 5 * N;
    S.fl1 = f32 + 6 * N; S.fl2 = f32 + 7 * N; S.fl3 = f32 + 8 * N; S.fb2 = f32 + 9 * N; S.fb3 = f32 + 10 * N;
    S.fw1 = f32 + 11 * N;
    S.rowbits = (uint32_t *)(smem + L.bits); S.colbits = S.rowbits + N2;
    S.Q = (uint32_t *)(smem + L.Q);
    S.rowid = (int *)(smem + L.rowid);
    S.red = (int2 *)(smem + L.red);
    S.wsum = (int *)(smem + L.wsum);
    int *qstart = S.wsum + 33, *pstart = qstart + 7;  // first entry of each pass, and the ends
    const int tid = threadIdx.x, bd = blockDim.x;
    const MeshDev &m = a.mesh;
    const PhononDev &P = a.ph;
    const Fc3Dev &fc = a.fc;
    const R *mwm = mwm_ptr<R>(fc);
    const C *egvs = egvs_ptr<C>(P);
    const int64_t ld = (int64_t)m.n_full * N;
    const int it = P.integrationtype;
    const float sigfix32 = (float)P.sigma_fixed;
    R *acc = (R *)(smem + L.total);  // ADJ with acc_in_smem: [fc.n * 27]
    int since_flush = 0;
    if constexpr (ADJ) {
        if (a.acc_in_smem)
            for (int i = tid; i < fc.n * 27; i += bd) acc[i] = (R)0;
    }

    // the next q-triplet's record is loaded one iteration ahead, so that the per-mode loads
    // of an iteration wait for one round trip to memory instead of two
    const int n_trip = a.n_trip_dev ? *a.n_trip_dev : a.n_trip;
    TripletRec rec_next = (int)blockIdx.x < n_trip ? a.trip[blockIdx.x] : TripletRec{};
    for (int t = blockIdx.x; t < n_trip; t += gridDim.x) {
        const TripletRec rec = rec_next;
        if (t + (int)gridDim.x < n_trip) rec_next = a.trip[t + gridDim.x];
        const int f1 = m.irr_full[rec.q1];
        const int q2 = rec.q2, q3 = rec.q3;
        const int i2 = m.full_irr[q2], i3 = m.full_irr[q3];
        const int nred = rec.red_cnt;
        const double perm = (q2 == q3) ? 1.0 : 2.0;
        // ---- what the screen reads: omega (NaN where no survivor may be: below 1e-9 Ha, or a
        // row that does not sample q2) and sigsq, FP32; -it 6: the widths of the mode pairs ----
        for (int i = tid; i < 3 * N; i += bd) {
            const int which = i / N, b = i - which * N;
            const int q = which == 0 ? f1 : (which == 1 ? q2 : q3);
            const float2 w = P.omega_hl[(size_t)q * N + b];
            bool on = true;
            if (which == 0) {
                const uint32_t mask = a.cand_mask[(size_t)rec.cand * 4 + (b >> 5)];
                const int r = (mask >> (b & 31)) & 1u ? a.rows.rowidx[(size_t)rec.q1 * N + b] : -1;
                S.rowid[b] = r;
                on = r >= 0;
            }
            f32[i] = on ? w.x : __int_as_float(0x7fc00000);
            f32[6 * N + i] = w.y;
            f32[3 * N + i] = P.sigsq32[(size_t)(which == 0 ? rec.q1 : (which == 1 ? i2 : i3)) * N + b];
        }
        if (it == 6)
            for (int i = tid; i < 3 * N2; i += bd) {
                const int which = i / N2, x = (i - which * N2) / N, y = i % N;
                W6[i] = adaptive_pair(P.vel + ((size_t)(which == 2 ? q2 : f1) * N + x) * 3,
                                      P.vel + ((size_t)(which == 0 ? q2 : q3) * N + y) * 3, P.reclat_g) / 3.0;
            }
        __syncthreads();
        const auto width6 = [&](int b1, int b2, int b3) {
            return W6[b1 * N + b2] + W6[N2 + b1 * N + b3] + W6[2 * N2 + b2 * N + b3] + P.thresh_sigma;
        };
        const auto width6_again = [&](int b1, int b2, int b3) {  // once A holds something else
            const double *v1 = P.vel + ((size_t)f1 * N + b1) * 3, *v2 = P.vel + ((size_t)q2 * N + b2) * 3,
                         *v3 = P.vel + ((size_t)q3 * N + b3) * 3;
            const double w12 = adaptive_pair(v1, v2, P.reclat_g) / 3.0, w13 = adaptive_pair(v1, v3, P.reclat_g) / 3.0;
            return w12 + w13 + adaptive_pair(v2, v3, P.reclat_g) / 3.0 + P.thresh_sigma;
        };
        // ---- screen: a thread per (b1, b2), its live bits kept in registers ----
        uint32_t live_lo = 0u, live_hi = 0u, live_x = 0u;  // 4 bits for b3 = 0..7, 8..15, 16..17
        int nsurv = 0;
        if (tid < N2) {
            const int b1 = tid / N, b2 = tid - b1 * N;
            const float o1 = S.fo1[b1], o2 = S.fo2[b2], l1 = S.fl1[b1], l2 = S.fl2[b2];
            const float s12 = S.fs1[b1] + S.fs2[b2], p12 = o1 + o2, d12 = o1 - o2;
            // |omega - omega'| < 1e-9 (scattering_threephonon.f90:90-101) where the high parts
            // are that near, decided on the pairs
            const float near1 = 1e-9f + 3e-7f * o1, near2 = 1e-9f + 3e-7f * o2;
            if (o1 == o1 && o2 == o2 && !close_f32(o1, l1, o2, l2)) {
#pragma unroll
                for (int b3 = 0; b3 < N; ++b3) {
                    const float o3 = S.fo3[b3];
                    float sg = sigfix32;
                    if (it == 2) sg = sqrt_screen(s12 + S.fs3[b3]);
                    else if (it == 6) sg = (float)width6(b1, b2, b3);
                    const float win = 8.0f * sg * 1.001f + 1e-6f * (p12 + o3);
                    uint32_t live = (fabsf(p12 - o3) <= win ? 1u : 0u) | (fabsf(d12 + o3) <= win ? 2u : 0u) |
                                    (fabsf(d12 - o3) <= win ? 4u : 0u) | (p12 + o3 <= win ? 8u : 0u);
                    if ((fabsf(o1 - o3) < near1 && close_f32(o1, l1, o3, S.fl3[b3])) ||
                        (fabsf(o2 - o3) < near2 && close_f32(o2, l2, o3, S.fl3[b3])))
                        live = 0u;
                    if (live) {
                        ++nsurv;
                        if (b3 < 8) live_lo |= live << (4 * b3);
                        else if (b3 < 16) live_hi |= live << (4 * (b3 - 8));
                        else live_x |= live << (4 * (b3 - 16));
                    }
                }
            }
        }
        // survivors in the low half, (b1, b2) with any in the high half (n^3 <= 5832 entries)
        int total = 0;
        const int off = block_exclusive_scan(nsurv | (nsurv ? 1 << 16 : 0), S.wsum, total);  // contains barriers
        if (total == 0) continue;
        // ---- the rest of the mode data, eigenvectors, equivalent triplets ----
        for (int b = tid; b < N; b += bd) {
            S.om1[b] = P.omega[(size_t)f1 * N + b];
            S.om2[b] = P.omega[(size_t)q2 * N + b];
            S.om3[b] = P.omega[(size_t)q3 * N + b];
            S.inv1[b] = P.inv_omega[(size_t)f1 * N + b];
            S.be2[b] = P.be[(size_t)i2 * N + b];
            S.be3[b] = P.be[(size_t)i3 * N + b];
            S.wrow[b] = a.rows.w3q[(size_t)rec.q1 * N + b];
            if constexpr (sizeof(R) == 8) {
                S.s1[b] = P.sigsq[(size_t)rec.q1 * N + b];
                S.s2[b] = P.sigsq[(size_t)i2 * N + b];
                S.s3[b] = P.sigsq[(size_t)i3 * N + b];
            } else {
                S.fb2[b] = (float)S.be2[b];
                S.fb3[b] = (float)S.be3[b];
                S.fw1[b] = (float)S.wrow[b];
            }
        }
        for (int i = tid; i < nred && i < kMaxRed; i += bd) S.red[i] = a.red[rec.red_off + i];
        for (int i = tid; i < 2 * N2; i += bd) S.rowbits[i] = 0u;
        for (int i = tid; i < 3 * N2; i += bd) {
            const int which = i / N2, e = i % N2;
            const int r = e / N, b = e % N;  // element (r) of mode b
            const int q = which == 0 ? f1 : (which == 1 ? q2 : q3);
            C *E = which == 0 ? E1 : (which == 1 ? E2 : E3);
            E[r * N + b] = egvs[((size_t)q * N + b) * N + r];
        }
        if (tid < N2) {
            const int b1 = tid / N;
            if (tid == b1 * N && b1 % NB1 == 0) {
                qstart[b1 / NB1] = off & 0xffff;
                pstart[b1 / NB1] = off >> 16;
            }
            if (nsurv) pairs[off >> 16] = (uint16_t)tid;
            if (tid == 0) {
                qstart[PASSES] = total & 0xffff;
                pstart[PASSES] = total >> 16;
            }
        }
        // ---- K2: pretransform into A ----
        int gi2[3], gi3[3];
        {
            const int n12 = m.grid[1] * m.grid[2];
            gi2[0] = q2 / n12; gi2[1] = (q2 / m.grid[2]) % m.grid[1]; gi2[2] = q2 % m.grid[2];
            gi3[0] = q3 / n12; gi3[1] = (q3 / m.grid[2]) % m.grid[1]; gi3[2] = q3 % m.grid[2];
            for (int d = 0; d < 3; ++d) {  // g_d L/N_d (phase3)
                gi2[d] *= m.lmul[d];
                gi3[d] *= m.lmul[d];
            }
        }
        constexpr int PC = phase_chunk(N, sizeof(C), ADJ);
        bool planned = false;
        if constexpr (sizeof(R) == 4) {
            // FP32 with a pretransform plan (all phase factors at once; k_threephonon_tc.cu
            // explains the plan): each thread's slots, 8 values and 8 words in flight, the
            // sums in the triplets' order as below; it writes the blocks that have triplets
            if (a.plan_slots > 0) {
                planned = true;
                for (int i = tid; i < N3; i += bd) A[i] = czero<C>();
                // four triplets per thread in flight: their lattice vectors, then their table entries
                for (int i0 = tid; i0 < fc.n + 4; i0 += 4 * bd) {
                    int kk[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int i = i0 + u * bd;
                        kk[u] = -1;
                        if (i < fc.n) {
                            const int32_t *lv = fc.lv + (size_t)i * 6;
                            int S2 = 0;
#pragma unroll
                            for (int d = 0; d < 3; ++d) S2 += gi2[d] * __ldg(lv + d) + gi3[d] * __ldg(lv + 3 + d);
                            int K = S2 % m.L;
                            kk[u] = K < 0 ? K + m.L : K;
                        }
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int i = i0 + u * bd;
                        if (i < fc.n + 4) ph[i] = kk[u] >= 0 ? twiddle_at<C>(fc, kk[u]) : czero<C>();
                    }
                }
                __syncthreads();
                const float4 *pm = a.plan_pm + tid;
                const uint32_t *pw = a.plan_word + tid;
                float ar = 0.f, ai = 0.f;
#pragma unroll 1
                for (int s0 = 0; s0 < a.plan_slots; s0 += 8) {
                    float4 mv[8];
                    uint32_t wd[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        mv[u] = __ldg(pm + (size_t)(s0 + u) * bd);
                        wd[u] = __ldg(pw + (size_t)(s0 + u) * bd);
                    }
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        const C *pp = ph + (wd[u] & 0xffffu);
                        const C p0 = pp[0], p1 = pp[1], p2 = pp[2], p3 = pp[3];
                        ar = fmaf(mv[u].x, p0.x, ar); ai = fmaf(mv[u].x, p0.y, ai);
                        ar = fmaf(mv[u].y, p1.x, ar); ai = fmaf(mv[u].y, p1.y, ai);
                        ar = fmaf(mv[u].z, p2.x, ar); ai = fmaf(mv[u].z, p2.y, ai);
                        ar = fmaf(mv[u].w, p3.x, ar); ai = fmaf(mv[u].w, p3.y, ai);
                        const uint32_t oc = wd[u] >> 16;  // on an element's last slot: its index + 1
                        if (oc) {
                            A[oc - 1u].x = ar;
                            A[oc - 1u].y = ai;
                            ar = 0.f;
                            ai = 0.f;
                        }
                    }
                }
            }
        }
        for (int c0 = 0; !planned && c0 < fc.n; c0 += PC) {
            const int cn = min(PC, fc.n - c0);
            if (c0) __syncthreads();
            for (int i = tid; i < cn; i += bd) ph[i] = phase3<C>(fc, m, gi2, gi3, c0 + i);
            __syncthreads();
            for (int idx = tid; idx < N3; idx += bd) {
                const int blk = idx / 27, ijk = idx % 27;
                const int lo = max(fc.blk_ptr[blk], c0), hi = min(fc.blk_ptr[blk + 1], c0 + cn);
                if (c0 && lo >= hi) continue;
                const int a1 = blk / (NA * NA), a2 = (blk / NA) % NA, a3 = blk % NA;
                const int ii = ijk % 3, jj = (ijk / 3) % 3, kk = ijk / 9;
                const int pa = 3 * a1 + ii, pb = 3 * a2 + jj, pc = 3 * a3 + kk;
                C *out = A + (pa * N + pb) * N + pc;
                C acc = c0 ? *out : czero<C>();
                for (int tt = lo; tt < hi; ++tt) {
                    const R mv = __ldg(mwm + (size_t)tt * 27 + ijk);
                    const C p = ph[tt - c0];
                    acc.x = fma(mv, p.x, acc.x);
                    acc.y = fma(mv, p.y, acc.y);
                }
                *out = acc;
            }
        }
        __syncthreads();
        // ---- the queue, in the phases' place: (b1 b2 b3) | live << 16 | place of (b1, b2) in
        // its pass << 20 ----
        const auto enqueue = [&]() {
            if (!nsurv) return;
            int k = off & 0xffff;
            const uint32_t place = (uint32_t)((off >> 16) - pstart[tid / N / NB1]) << 20;
#pragma unroll
            for (int b3 = 0; b3 < N; ++b3) {
                const uint32_t live = b3 < 8 ? (live_lo >> (4 * b3)) & 15u
                                             : (b3 < 16 ? (live_hi >> (4 * (b3 - 8))) & 15u : (live_x >> (4 * (b3 - 16))) & 15u);
                if (live) S.Q[k++] = (uint32_t)(tid * N + b3) | (live << 16) | place;
            }
        };
        if constexpr (!ADJ) enqueue();
        // ---- K3: T1 in place (a thread owns a column) ----
        if (tid < N2) {
            const int bc = tid;
            C acc[N];
#pragma unroll
            for (int b1 = 0; b1 < N; ++b1) acc[b1] = czero<C>();
#pragma unroll 3
            for (int aa = 0; aa < N; ++aa) {
                const C p = A[aa * N2 + bc];
#pragma unroll
                for (int b1 = 0; b1 < N; ++b1) cfma(acc[b1], E1[aa * N + b1], p);
            }
#pragma unroll
            for (int b1 = 0; b1 < N; ++b1) A[b1 * N2 + bc] = acc[b1];
        }
        __syncthreads();
        for (int pass = 0; pass < PASSES; ++pass) {
            // T2[place][c] of the pass's pairs into B
            const int p0 = pstart[pass], np = pstart[pass + 1] - p0;
            for (int i = tid; i < np * N; i += bd) {
                const int k = i / N, c = i - k * N, pr = pairs[p0 + k], b1 = pr / N, b2 = pr - b1 * N;
                const C *t1 = A + b1 * N2 + c, *e = E2 + b2;
                C acc = czero<C>();
#pragma unroll
                for (int b = 0; b < N; ++b) cfma(acc, e[b * N], t1[b * N]);
                B[i] = acc;
            }
            __syncthreads();
            // Psi, delta weights and occupations of the pass's survivors; the forward pass writes F
            // over T1 of its b1 (dense, read only where the row/column bits are set)
            C psi;
            const auto contract = [&](uint32_t qv) {
                const C *t2 = B + (qv >> 20) * N, *e = E3 + (qv & 0xffffu) % N;
                psi = czero<C>();
#pragma unroll
                for (int c = 0; c < N; ++c) cfma(psi, e[c * N], t2[c]);
            };
            if constexpr (!ADJ) {
                const auto put = [&](uint32_t qv, R f) {
                    const int idx = (int)(qv & 0xffffu), b1 = idx / N2;
                    F[b1 * FS + (idx - b1 * N2)] = (double)f;
                    if (f != (R)0) k3_mark<N>(S, idx);
                };
                const auto psisq = [&](uint32_t qv) -> R {
                    contract(qv);
                    return psi.x * psi.x + psi.y * psi.y;
                };
                if constexpr (sizeof(R) == 8)
                    k3_survivors<N>(S, P, qstart[pass], qstart[pass + 1], perm, width6, psisq, put);
                else
                    k3_survivors_f32<N, true>(S, P, qstart[pass], qstart[pass + 1], (float)perm, width6, psisq, put);
                if (pass + 1 < PASSES) __syncthreads();  // B and the next T1 slabs
            } else {
                // d L / d|Psi_b|^2 = lam[row(b1)] * nred * dF_b/d|Psi_b|^2 (Gamma += nred * sum F);
                // d|Psi|^2 / d P[abc] = 2 Re(conj(Psi) E1[a][b1] E2[b][b2] E3[c][b3]), so with
                // W = G conj(Psi):  Q[abc] = sum_b W_b E1[a][b1] E2[b][b2] E3[c][b3] and
                // d L / d mwm_t(i,j,k) = 2 Re(phase_t Q[3a1+i][3a2+j][3a3+k]).
                // with a scattering-matrix cotangent xi_bar (the BTE adjoint): the Xi row terms
                // 2 F om2/om1 at (q2', b2) and 2 F om3/om1 at (q3', b3) of every equivalent
                // triplet add xi_bar(row, .) times those factors to the cotangent of F;
                // R2[b1][b2] and XB[b1][b3] hold xi_bar summed over the equivalent triplets
                double *XB = (double *)(smem + L.xb);
                if (a.xi_bar)
                    for (int e = tid; e < 2 * N2; e += bd) {
                        const int x = e % N2, b1 = x / N, bb = x % N, row = S.rowid[b1];
                        double sum = 0.0;
                        if (row >= 0) {
                            const double *wr = a.xi_bar + (int64_t)row * ld;
                            for (int k = 0; k < nred; ++k) {
                                const int2 pr = S.red[k];
                                sum += wr[(int64_t)(e < N2 ? pr.x : pr.y) * N + bb];
                            }
                        }
                        if (e < N2) S.R2[x] = sum;
                        else XB[x] = sum;
                    }
                for (int i = tid; i < N3; i += bd) A[i] = czero<C>();
                enqueue();
                __syncthreads();
                const auto psisq = [&](uint32_t qv) -> R {  // F without |Psi|^2, and Psi
                    contract(qv);
                    return (R)1;
                };
                const auto put = [&](uint32_t qv, R f) {
                    const int idx = (int)(qv & 0xffffu), b1 = idx / N2, row = S.rowid[b1];
                    double cot = a.lam[row] * (double)nred;
                    if (a.xi_bar) {
                        const int b2 = (idx / N) % N, b3 = idx % N;
                        cot += 2.0 * (S.om2[b2] * S.R2[b1 * N + b2] + S.om3[b3] * XB[b1 * N + b3]) * S.inv1[b1];
                    }
                    const double g = cot * (double)f;
                    C w;
                    w.x = (R)(g * (double)psi.x);
                    w.y = (R)(-g * (double)psi.y);
                    A[idx] = w;
                };
                if constexpr (sizeof(R) == 8)
                    k3_survivors<N>(S, P, qstart[pass], qstart[pass + 1], perm, width6_again, psisq, put);
                else
                    k3_survivors_f32<N, true>(S, P, qstart[pass], qstart[pass + 1], (float)perm, width6_again, psisq, put);
            }
        }
        if constexpr (ADJ) {
            __syncthreads();
            // the queue took the place of two of the eigenvector matrices: load them again
            for (int i = tid; i < 2 * N2; i += bd) {
                const int e = i % N2;
                (i < N2 ? E1 : E2)[e] = egvs[((size_t)(i < N2 ? f1 : q2) * N + e % N) * N + e / N];
            }
            __syncthreads();
            if (tid < N2) {  // B[a][b2b3] = sum_b1 E1[a][b1] W[b1][b2b3]
                const int bc = tid;
                C acc[N];
#pragma unroll
                for (int x = 0; x < N; ++x) acc[x] = czero<C>();
#pragma unroll 3
                for (int b1 = 0; b1 < N; ++b1) {
                    const C w = A[b1 * N2 + bc];
#pragma unroll
                    for (int x = 0; x < N; ++x) cfma(acc[x], E1[x * N + b1], w);
                }
#pragma unroll
                for (int x = 0; x < N; ++x) B[x * N2 + bc] = acc[x];
            }
            __syncthreads();
            if (tid < N2) {  // A[a][b][b3] = sum_b2 E2[b][b2] B[a][b2][b3]
                const int aa = tid / N, b3 = tid % N;
                C acc[N];
#pragma unroll
                for (int x = 0; x < N; ++x) acc[x] = czero<C>();
#pragma unroll 3
                for (int b2 = 0; b2 < N; ++b2) {
                    const C tv = B[(aa * N + b2) * N + b3];
#pragma unroll
                    for (int x = 0; x < N; ++x) cfma(acc[x], E2[x * N + b2], tv);
                }
#pragma unroll
                for (int x = 0; x < N; ++x) A[(aa * N + x) * N + b3] = acc[x];
            }
            __syncthreads();
            if (tid < N2) {  // B[a][b][c] = sum_b3 E3[c][b3] A[a][b][b3]
                const int ab = tid;
                C acc[N];
#pragma unroll
                for (int x = 0; x < N; ++x) acc[x] = czero<C>();
#pragma unroll 3
                for (int b3 = 0; b3 < N; ++b3) {
                    const C tv = A[ab * N + b3];
#pragma unroll
                    for (int x = 0; x < N; ++x) cfma(acc[x], E3[x * N + b3], tv);
                }
#pragma unroll
                for (int x = 0; x < N; ++x) B[ab * N + x] = acc[x];
            }
            // the CTA's slice: doubles on the FP64 path, floats on the mixed path (contiguous
            // slices of n_fc3 * 27 entries of either type)
            double *slice = a.mwm_bar + (size_t)blockIdx.x * fc.n * 27;
            float *slicef = reinterpret_cast<float *>(a.mwm_bar) + (size_t)blockIdx.x * fc.n * 27;
            // thread -> one (i,j,k) of the 27 and every groups-th force-constant triplet; within a
            // q-triplet exactly one thread touches each entry, and q-triplets are separated by
            // barriers
            const int groups = bd / 27, grp = tid / 27, ijk = tid % 27;
            const int off3 = (ijk % 3) * N2 + ((ijk / 3) % 3) * N + ijk / 9;
            constexpr int PCA = phase_chunk(N, sizeof(C), ADJ);
            for (int c0 = 0; c0 < fc.n; c0 += PCA) {
                const int cn = min(PCA, fc.n - c0);
                __syncthreads();
                for (int i = tid; i < cn; i += bd) ph[i] = phase3<C>(fc, m, gi2, gi3, c0 + i);
                __syncthreads();
                if (grp < groups) {
                    for (int tl = grp; tl < cn; tl += groups) {
                        const int tt = c0 + tl;
                        const C q = B[fc.abase[tt] + off3];
                        const C p = ph[tl];
                        const R v = (R)2 * (p.x * q.x - p.y * q.y);
                        if (a.acc_in_smem) {
                            acc[(size_t)tt * 27 + ijk] += v;
                        } else if constexpr (sizeof(R) == 8) {
                            slice[(size_t)tt * 27 + ijk] += (double)v;
                        } else {
                            slicef[(size_t)tt * 27 + ijk] += (float)v;
                        }
                    }
                }
            }
            __syncthreads();
            if (a.acc_in_smem && ++since_flush == kAdjFlush) {
                for (int i = tid; i < fc.n * 27; i += bd) {
                    if constexpr (sizeof(R) == 8)
                        slice[i] += (double)acc[i];
                    else
                        slicef[i] += (float)acc[i];
                    acc[i] = (R)0;
                }
                since_flush = 0;
                __syncthreads();
            }
            continue;
        }
        // ---- R2 = sum over b3, R3 = sum over b2 (into B as doubles), Gamma and Xi ----
        k3_sums_scatter<N, false, FS>(S, a, nred);
    }
    if constexpr (ADJ) {
        if (a.acc_in_smem) {
            __syncthreads();
            double *slice = a.mwm_bar + (size_t)blockIdx.x * fc.n * 27;
            float *slicef = reinterpret_cast<float *>(a.mwm_bar) + (size_t)blockIdx.x * fc.n * 27;
            for (int i = tid; i < fc.n * 27; i += bd) {
                if constexpr (sizeof(R) == 8)
                    slice[i] += (double)acc[i];
                else
                    slicef[i] += (float)acc[i];
            }
        }
    }
}

// Persistent grid: resident CTAs per SM times the SM count, at most one CTA per item.
// `extra` bytes of dynamic shared memory follow the kernel's layout (adjoint accumulator).
template <int N, typename R, bool ADJ>
int grid_n(int n_sm, int n_trip, size_t extra, int ctas_per_sm = 0, int *api = nullptr, int *count = nullptr) {
    const Layout L = make_layout(N, sizeof(typename CT<R>::C), ADJ);
    const size_t bytes = L.total + extra;
    int per_sm = resident_ctas((const void *)k_threephonon<N, R, ADJ>, threads_for(N), bytes, api, count);
    if (per_sm < 1) return 0;
    if (ctas_per_sm > 0 && ctas_per_sm < per_sm) per_sm = ctas_per_sm;
    const int grid = n_sm * per_sm;
    return grid > n_trip ? (n_trip > 0 ? n_trip : 1) : grid;
}

template <int N, typename R, bool ADJ>
cudaError_t launch_grid(const ThreePhArgs &a, int grid, size_t extra, cudaStream_t s) {
    const Layout L = make_layout(N, sizeof(typename CT<R>::C), ADJ);
    k_threephonon<N, R, ADJ><<<grid, threads_for(N), L.total + extra, s>>>(a);
    return cudaGetLastError();
}

template <int N, typename R>
cudaError_t launch_n(const ThreePhArgs &a, int n_sm, int ctas_per_sm, cudaStream_t s) {
    const int grid = grid_n<N, R, false>(n_sm, a.n_trip, 0, ctas_per_sm);
    if (grid < 1) return cudaErrorInvalidConfiguration;
    return launch_grid<N, R, false>(a, grid, 0, s);
}

template <typename R, bool ADJ>
int grid_prec(int n, int n_sm, int n_trip, size_t extra, int *api = nullptr, int *count = nullptr) {
    switch (n) {
        case 3: return grid_n<3, R, ADJ>(n_sm, n_trip, extra, 0, api, count);
        case 6: return grid_n<6, R, ADJ>(n_sm, n_trip, extra, 0, api, count);
        case 9: return grid_n<9, R, ADJ>(n_sm, n_trip, extra, 0, api, count);
        case 12: return grid_n<12, R, ADJ>(n_sm, n_trip, extra, 0, api, count);
        case 15: return grid_n<15, R, ADJ>(n_sm, n_trip, extra, 0, api, count);
        case 18: return grid_n<18, R, ADJ>(n_sm, n_trip, extra, 0, api, count);
        default: return 0;
    }
}

template <typename R>
cudaError_t launch_adj_prec(const ThreePhArgs &a, int grid, size_t extra, cudaStream_t s) {
    switch (a.mesh.n_mode) {
        case 3: return launch_grid<3, R, true>(a, grid, extra, s);
        case 6: return launch_grid<6, R, true>(a, grid, extra, s);
        case 9: return launch_grid<9, R, true>(a, grid, extra, s);
        case 12: return launch_grid<12, R, true>(a, grid, extra, s);
        case 15: return launch_grid<15, R, true>(a, grid, extra, s);
        case 18: return launch_grid<18, R, true>(a, grid, extra, s);
        default: return cudaErrorNotSupported;
    }
}

// The q-triplets with a mode triplet inside an 8-sigma window: a thread per q-triplet, the
// screen of k_threephonon (a superset of it: no degeneracy rules, the windows compared as
// squares) to the first hit. The fused kernel spends a CTA's loads and barriers on every
// q-triplet before it knows that nothing survives, and 76 % of rocksalt 24^3 are such: device time of
// the call 7.5..8.0 -> 5.2 ms (2.0 million q-triplets, mixed).
template <int N>
__global__ void __launch_bounds__(128) k_threephonon_prescreen(ThreePhArgs a, TripletRec *live, int32_t *count) {
    const int t = blockIdx.x * 128 + threadIdx.x, lane = threadIdx.x & 31;
    const PhononDev &P = a.ph;
    const MeshDev &m = a.mesh;
    bool any = false;
    TripletRec rec{};
    if (t < a.n_trip) {
        rec = a.trip[t];
        const uint32_t mask = a.cand_mask[(size_t)rec.cand * 4];
        const float2 *w1 = P.omega_hl + (size_t)m.irr_full[rec.q1] * N, *w2 = P.omega_hl + (size_t)rec.q2 * N,
                     *w3 = P.omega_hl + (size_t)rec.q3 * N;
        const bool fixed = P.integrationtype == 1;
        const float *g1 = P.sigsq32 + (size_t)rec.q1 * N, *g2 = P.sigsq32 + (size_t)m.full_irr[rec.q2] * N,
                    *g3 = P.sigsq32 + (size_t)m.full_irr[rec.q3] * N;
        // 64.2 > (8 * 1.001)^2; a fixed width counts once
        const float sf = fixed ? 64.2f * (float)P.sigma_fixed * (float)P.sigma_fixed : 0.f, sc = fixed ? 0.f : 64.2f;
        float o2[N], o3[N], s2[N], s3[N];
#pragma unroll
        for (int b = 0; b < N; ++b) {
            o2[b] = w2[b].x;
            o3[b] = w3[b].x;
            s2[b] = sc * g2[b];
            s3[b] = sc * g3[b] + sf;
        }
        for (int b1 = 0; b1 < N && !any; ++b1) {
            const float o1 = w1[b1].x, s1 = sc * g1[b1];
            // NaN (omega below 1e-9 Ha) fails every comparison
            if (!((mask >> b1) & 1u) || a.rows.rowidx[(size_t)rec.q1 * N + b1] < 0 || o1 != o1) continue;
#pragma unroll
            for (int b2 = 0; b2 < N; ++b2) {
                const float p = o1 + o2[b2], d = o1 - o2[b2], s12 = s1 + s2[b2];
#pragma unroll
                for (int b3 = 0; b3 < N; ++b3) {
                    // om1 + om2 + om3 is never the smallest of the four mismatches
                    const float x = fminf(fminf(fabsf(p - o3[b3]), fabsf(d + o3[b3])), fabsf(d - o3[b3])) -
                                    1e-6f * (p + o3[b3]);
                    any |= x <= 0.f || x * x <= s12 + s3[b3];
                }
            }
        }
    }
    const uint32_t bal = __ballot_sync(0xffffffffu, any);
    int at = 0;
    if (lane == 0 && bal) at = atomicAdd(count, __popc(bal));
    at = __shfl_sync(0xffffffffu, at, 0);
    if (any) live[at + __popc(bal & ((1u << lane) - 1u))] = rec;
}

constexpr int64_t kPrescreen6 = 16384, kPrescreen3 = 1 << 20;

// Sums of n_slice slices of `pitch` entries, 32 entries and 8 groups of slices per block (one
// thread per entry had left most of the chip idle, and its FP64 additions bound it: 73 us for
// 456 slices of 30 105 entries). Slices in FP32 are summed in double-float (exact to ~2^-44),
// the groups in FP64. Quads: entry [ijk][triplet] of the tensor-core adjoint, the triplets padded
// to a multiple of four, goes to out[27 triplet + ijk].
template <typename T, bool Quads>
__global__ void __launch_bounds__(256) k_sum_slices(const T *slices, int32_t n_slice, int64_t pitch, int32_t n_fc,
                                                    double *out) {
    __shared__ double part[8][33];
    const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
    const int64_t e = (int64_t)blockIdx.x * 32 + x;
    double acc = 0.0;
    if (e < pitch) {
        if constexpr (sizeof(T) == sizeof(float)) {
            float2 s = make_float2(0.f, 0.f);
#pragma unroll 8
            for (int g = y; g < n_slice; g += 8) df_acc(s, slices[(int64_t)g * pitch + e]);
            acc = (double)s.x + (double)s.y;
        } else {
#pragma unroll 4
            for (int g = y; g < n_slice; g += 8) acc += slices[(int64_t)g * pitch + e];
        }
    }
    part[y][x] = acc;
    __syncthreads();
    if (y != 0 || e >= pitch) return;
    for (int k = 1; k < 8; ++k) acc += part[k][x];
    if constexpr (Quads) {
        const int64_t n4 = pitch / 27, t = e % n4;
        if (t < n_fc) out[t * 27 + e / n4] = acc;
    } else {
        out[e] = acc;
    }
}

template <typename R>
cudaError_t launch_prec(const ThreePhArgs &a, int n_sm, int ctas_per_sm, cudaStream_t s) {
    switch (a.mesh.n_mode) {
        case 3: return launch_n<3, R>(a, n_sm, ctas_per_sm, s);
        case 6: return launch_n<6, R>(a, n_sm, ctas_per_sm, s);
        case 9: return launch_n<9, R>(a, n_sm, ctas_per_sm, s);
        case 12: return launch_n<12, R>(a, n_sm, ctas_per_sm, s);
        case 15: return launch_n<15, R>(a, n_sm, ctas_per_sm, s);
        case 18: return launch_n<18, R>(a, n_sm, ctas_per_sm, s);
        default: return cudaErrorNotSupported;
    }
}

}  // namespace

namespace {
__global__ void k_exp_neg_check(const double *t, int32_t n, double *out, const double *tab) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = exp_neg(t[i], tab);
}
}  // namespace

cudaError_t launch_exp_neg_check(const double *t, int32_t n, double *out, const double *tab, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    k_exp_neg_check<<<(n + 255) / 256, 256, 0, s>>>(t, n, out, tab);
    return cudaGetLastError();
}

int threephonon_threads(int n) { return threads_for(n); }

bool threephonon_plan_fits(int n, int n_fc) {
    // the plan path holds all phase factors (and 4 zero ones after them) in the phase region
    return n >= 3 && n <= 16 && n_fc + 4 <= phase_chunk(n, (int)sizeof(float2), true);
}

size_t threephonon_smem_bytes(int n, int precision, int) {
    return make_layout(n, precision == 0 ? sizeof(double2) : sizeof(float2)).total;
}

// From 9 modes on nearly all q-triplets have a survivor (12 modes, 9^3: 99 %; 15 modes, 8^3: 99 %),
// and width type 6 is not screened by squares. Device time of the call in us, without and with
// the pass:
//   6 modes, adaptive  3 260 q-triplets (42 % left): FP64 246, 214; mixed 158, 153
//                     11 620 (37 %): 426, 374; 210, 180.  33 490 (33 %): 804, 710; 325, 264
//                    181 902 (29 %): 3031, 2750; 984, 731.  2.0 million (24 %): 24 640, 23 800; 7745, 5190
//   6 modes, one width  3 260 (85 %): 290, 290; 159, 165.  33 490 (85 %): 1657, 1564; 418, 395
//   3 modes, adaptive 82 611 (48 %): 894, 884; 432, 436.  365 333 (43 %): 3250, 3250; 1400, 1428
//                      2.0 million (39 %): 15 790, 15 000; 6790, 6490
//   3 modes, one width, none left out: 82 611: 1721, 1718; 790, 797
// so at 6 modes from some 16 000 q-triplets on, at 3 modes, where the fused kernel's loads and
// barriers are few, with adaptive widths from a million on.
bool threephonon_prescreen_for(int n, int integrationtype, int64_t n_trip) {
    if (n == 6) return integrationtype != 6 && n_trip >= kPrescreen6;
    return n == 3 && integrationtype == 2 && n_trip >= kPrescreen3;
}

cudaError_t launch_threephonon_prescreen(const ThreePhArgs &a, TripletRec *live, int32_t *count, cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(count, 0, sizeof(int32_t), s);
    if (e != cudaSuccess || a.n_trip <= 0) return e;
    const unsigned grid = (unsigned)((a.n_trip + 127) / 128);
    switch (a.mesh.n_mode) {
        case 3: k_threephonon_prescreen<3><<<grid, 128, 0, s>>>(a, live, count); break;
        case 6: k_threephonon_prescreen<6><<<grid, 128, 0, s>>>(a, live, count); break;
        default: return cudaErrorNotSupported;
    }
    return cudaGetLastError();
}

cudaError_t launch_threephonon(const ThreePhArgs &a, int precision, int n_sm, int ctas_per_sm, cudaStream_t s) {
    if (a.n_trip <= 0) return cudaSuccess;
    if (precision == 0) return launch_prec<double>(a, n_sm, ctas_per_sm, s);
    return launch_prec<float>(a, n_sm, ctas_per_sm, s);
}

int threephonon_max_per_sm(int n, int precision, int *api, int *count) {
    // grid_n with one SM and an unbounded item count gives the CTAs that fit on one SM
    return precision == 0 ? grid_prec<double, false>(n, 1, 1 << 30, 0, api, count)
                          : grid_prec<float, false>(n, 1, 1 << 30, 0, api, count);
}

int threephonon_adjoint_grid(int n, int precision, int n_sm, int n_trip, int n_fc, bool acc_in_smem) {
    const size_t extra = acc_in_smem ? (size_t)n_fc * 27 * (precision == 0 ? sizeof(double) : sizeof(float)) : 0;
    return precision == 0 ? grid_prec<double, true>(n, n_sm, n_trip, extra)
                          : grid_prec<float, true>(n, n_sm, n_trip, extra);
}

cudaError_t launch_threephonon_adjoint(const ThreePhArgs &a, int precision, int grid, cudaStream_t s) {
    if (a.n_trip <= 0 || grid <= 0) return cudaSuccess;
    const size_t extra =
        a.acc_in_smem ? (size_t)a.fc.n * 27 * (precision == 0 ? sizeof(double) : sizeof(float)) : 0;
    if (precision == 0) return launch_adj_prec<double>(a, grid, extra, s);
    return launch_adj_prec<float>(a, grid, extra, s);
}

cudaError_t launch_sum_slices(const double *slices, int32_t n_slice, int32_t n_fc, bool quads, int precision,
                              double *out, cudaStream_t s) {
    const int64_t pitch = adjoint_slice_entries(n_fc, quads);
    if (pitch <= 0) return cudaSuccess;
    const unsigned g = (unsigned)((pitch + 31) / 32);
    const float *f = reinterpret_cast<const float *>(slices);
    if (quads)
        k_sum_slices<float, true><<<g, 256, 0, s>>>(f, n_slice, pitch, n_fc, out);
    else if (precision == 0)
        k_sum_slices<double, false><<<g, 256, 0, s>>>(slices, n_slice, pitch, n_fc, out);
    else
        k_sum_slices<float, false><<<g, 256, 0, s>>>(f, n_slice, pitch, n_fc, out);
    return cudaGetLastError();
}

}  // namespace tdg
