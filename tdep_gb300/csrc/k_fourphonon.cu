// Fused four-phonon scattering for one accepted irreducible q-quartet per CTA iteration
// (persistent grid-stride loop over the quartet list).
//
// Reference (src/thermal_conductivity/scattering_fourphonon.f90):
//   pretransform_phi4 (:459-506)  ptf(a,b,c,d) = sum_t mwm_t(i,j,k,l) exp(-2 pi i (q2.lv2 + q3.lv3 + q4.lv4))
//   zgeru x3 + dot_product (:131-159)  c0 = sum_abcd e1(a) e2(b) e3(c) e4(d) ptf(a,b,c,d)
//   get_dirac (:267-327), multiplicities (:104-122), accumulation (:161-186).
// The reference rebuilds the n^4 ptf per row and contracts it per (b2,b3,b4) (2 n^4
// complex MACs per mode quadruplet, n^8 per row). Here, per q-quartet:
//   T1[b1][b][c][d] = sum_a E1[a][b1] ptf[a][b][c][d], ptf = sum_t mwm_t(i,j,k,l) phase_t
// is built once for every row mode b1 into a per-CTA slice of device scratch: first the
// pretransform ptf (n_fc4 * 81 real x complex MACs), then its contraction with E1 in place
// (n^5 complex MACs); for each row b1 the n^3 slice of T1 is contracted with E2, E3, E4 in
// shared memory (3 n^4 complex MACs per b1): 4 n^5 complex MACs per q-quartet in all.
// Phases are exact roots of unity from integer lattice vectors, as in the three-phonon
// kernel.
//   The delta weights. 13 to 40 % of the mode quadruplets have a Gaussian inside its 8-sigma
// window with adaptive widths, so an FP32 screen with a safety margin (a Gaussian it drops is
// exactly zero in the reference) queues them, and full warps contract the last index (E4) for
// the queued ones alone and form their weights. Precision R: double (FP64 path: weights,
// occupations and accumulation in FP64 with the reference's window test) or float (mixed
// path: FP32 pretransform, contraction, weights and occupations; the centre differences from
// FP32 frequency pairs and the sums over modes in double-float, so that nothing per
// quadruplet touches the FP64 pipe, which at 2 lanes per clock and SM was 83 % of this
// kernel's time with FP64 centre differences and conversions).
//   Measured: perovskite 8^3, 27 x 27 pairs, mixed 4.18 -> 1.75 ms (issue and shared-memory
// bound); rocksalt 8^3 FP64 1.13 -> 0.79 ms (91 % of the FP64 pipe).
#include <cuda_runtime.h>

#include <type_traits>

#include "dev_common.cuh"
#include "tdg_internal.cuh"

namespace tdg {

namespace {

constexpr double kFourPhononPrefactor = 3.141592653589793 / 96.0;
// Phase factors at a time: those of one leading atom at once where that costs no CTA (519 of
// the five-atom perovskite; a second pass reads and writes every output again).
__host__ __device__ constexpr int phase_chunk4(int n) { return n >= 12 ? 1024 : 512; }

// Modes b1 that go through the second to fourth stage together: few modes leave most of a
// CTA idle between barriers.
__host__ __device__ constexpr int b1_batch(int n) { return n <= 6 ? n : (n <= 9 ? 3 : 1); }
// From 12 modes on a thread owns a column of the second and third stage (n outputs from n
// inputs in registers), in place; below, n^2 columns are too few and a thread takes one output.
__host__ __device__ constexpr bool by_column(int n) { return n >= 12; }

template <typename R>
__device__ __forceinline__ const R *mwm4_ptr(const Fc4Dev &fc);
template <>
__device__ __forceinline__ const double *mwm4_ptr<double>(const Fc4Dev &fc) {
    return fc.mwm;
}
template <>
__device__ __forceinline__ const float *mwm4_ptr<float>(const Fc4Dev &fc) {
    return fc.mwm32;
}

template <typename C>
__device__ __forceinline__ C twiddle4(const FourPhArgs &a, int k);
template <>
__device__ __forceinline__ double2 twiddle4<double2>(const FourPhArgs &a, int k) {
    return a.twiddle[k];
}
template <>
__device__ __forceinline__ float2 twiddle4<float2>(const FourPhArgs &a, int k) {
    return a.twiddle32[k];
}

template <typename C>
__device__ __forceinline__ const C *egvs4_ptr(const PhononDev &ph);
template <>
__device__ __forceinline__ const double2 *egvs4_ptr<double2>(const PhononDev &ph) {
    return ph.egvs;
}
template <>
__device__ __forceinline__ const float2 *egvs4_ptr<float2>(const PhononDev &ph) {
    return ph.egvs32;
}

struct Layout4 {
    size_t om, be, sg, fo, inv1, wrow, rowid, red, R, occ, E, ph, Q, w6, A, B, F, total;
};
__host__ __device__ inline size_t al16(size_t x) { return (x + 15) & ~size_t(15); }
// it6: with the width tables of -it 6.
__host__ __device__ inline Layout4 make_layout4(int n, int cs, bool it6) {
    Layout4 L;
    size_t o = 0;
    const size_t n2 = (size_t)n * n, n3 = n2 * n, nb = b1_batch(n), rs = cs / 2;
    L.om = o; o += al16(sizeof(double) * 4 * n);     // omega of q1..q4
    L.be = o; o += al16(sizeof(double) * 4 * n);     // Bose factors of q2..q4 (slot 0 unused)
    L.sg = o; o += al16(sizeof(double) * 4 * n);     // sigsq of q1..q4
    L.fo = o; o += al16(sizeof(float) * 12 * n);     // omega, sigsq and omega's rest in FP32
    L.inv1 = o; o += al16(sizeof(double) * n);
    L.wrow = o; o += al16(sizeof(double) * n);
    L.rowid = o; o += al16(sizeof(int) * (n + 4));   // and the queue's length
    L.red = o; o += al16(sizeof(int4) * kMaxRed);
    L.R = o; o += al16(sizeof(double) * 4 * n * nb);
    L.occ = o; o += al16(rs * (2 * n2 + 6 * n));     // occupation products (see below)
    L.E = o; o += al16((size_t)cs * 4 * n2);
    // the phases, then the survivor queue, then the sums over one mode (2 n^2 per b1)
    const size_t phz = (size_t)cs * phase_chunk4(n), qz = sizeof(uint32_t) * nb * n3, xz = sizeof(double) * 2 * nb * n2;
    L.ph = L.Q = o;
    o += al16(phz > qz ? (phz > xz ? phz : xz) : (qz > xz ? qz : xz));
    L.w6 = o; o += it6 ? al16(sizeof(double) * 6 * n2) : 0;
    L.A = o; o += al16(cs * nb * n3);
    L.B = o; o += by_column(n) ? 0 : al16(cs * nb * n3);
    L.F = o; o += al16(rs * nb * n3);
    L.total = o;
    return L;
}

__host__ __device__ constexpr int threads4_for(int n) { return n >= 9 ? 256 : ((n * n * n + 31) / 32) * 32; }

// Resident CTAs the register budget is sized for: what shared memory admits (1 at 15 modes in
// FP64, 2 at 9 and 12).
__host__ __device__ constexpr int min_blocks4(int n, bool dbl) {
    return n <= 3 ? 16 : (n <= 6 ? 3 : (dbl ? (n <= 12 ? 2 : 1) : 3));
}

// om1 - (m2 + m3 + m4) from FP32 pairs omega = h + l, as centre_diff_f32 for three.
__device__ __forceinline__ float centre_diff4_f32(float h1, float l1, float h2, float l2, float h3, float l3, float h4,
                                                  float l4) {
    const float s = h2 + h3, bs = s - h2;
    const float es = (h2 - (s - bs)) + (h3 - bs);
    const float u = s + h4, bu = u - s;
    const float eu = (s - (u - bu)) + (h4 - bu);
    const float d = h1 - u, bd = d - h1;
    const float ed = (h1 - (d - bd)) + (-u - bd);
    return d + (ed + ((l1 - l2 - l3 - l4) - (es + eu)));
}

// The eight Gaussians of get_dirac (scattering_fourphonon.f90:267-327), centred at +-om2 +-om3
// +-om4: bit j of these is set where the sign is plus. d[j / 2] = g(even j) - g(odd j).
constexpr uint32_t kPlus2 = 0x59u, kPlus3 = 0x65u, kPlus4 = 0x95u;

template <int N, typename R>
__global__ void __launch_bounds__(threads4_for(N), min_blocks4(N, sizeof(R) == 8)) k_fourphonon(FourPhArgs a) {
    using C = typename CT<R>::C;
    constexpr int N2 = N * N, N3 = N2 * N, NB = b1_batch(N);
    constexpr int NA = N / 3;
    constexpr bool DBL = sizeof(R) == 8, COLS = by_column(N);
    static_assert(N % NB == 0 && (!COLS || NB == 1), "batches of b1");
    extern __shared__ __align__(16) unsigned char smem[];
    const PhononDev &P = a.ph;
    const int it = P.integrationtype;
    const Layout4 L = make_layout4(N, sizeof(C), it == 6);
    double *om = (double *)(smem + L.om);   // om[k*N + b], k = 0..3 for q1..q4
    double *be = (double *)(smem + L.be);
    double *sg = (double *)(smem + L.sg);
    float *fo = (float *)(smem + L.fo);     // fo[k*N + b] omega, fo[(4+k)*N + b] sigsq, fo[(8+k)*N + b] omega's rest
    double *inv1 = (double *)(smem + L.inv1);
    double *wrow = (double *)(smem + L.wrow);
    int *rowid = (int *)(smem + L.rowid), *qlen = rowid + N;
    int4 *red = (int4 *)(smem + L.red);
    // the row terms 2 R om / om1 of R2, R3, R4 (sums over the other two modes) for each b1 of
    // the batch, then R2 itself
    double *Rs = (double *)(smem + L.R), *R2 = Rs + 3 * N * NB;
    // Occupation products of the quartet, so that the four polynomials of the weights
    // (scattering_fourphonon.f90:161-186) cost 10 operations per mode quadruplet instead of
    // 26: per (b3, b4) P00 = n3 n4 and P11 = (n3+1)(n4+1), with n3 (n4+1) = P00 + n3 and
    // (n3+1) n4 = P00 + n4; per b2 n2, n2+1, 3 n2, 3 (n2+1). Formed in FP64, kept in R.
    R *P00 = (R *)(smem + L.occ), *P11 = P00 + N2;
    R *N2v = P11 + N2, *N2p = N2v + N, *N2x3 = N2p + N, *N2px3 = N2x3 + N, *N3v = N2px3 + N, *N4v = N3v + N;
    C *E = (C *)(smem + L.E);               // E[k*N2 + r*N + b], k = 0..3
    C *ph = (C *)(smem + L.ph);
    uint32_t *Q = (uint32_t *)(smem + L.Q); // (b1 b2 b3 b4) within the batch | live Gaussians << 16
    double *W6d = (double *)(smem + L.w6);  // -it 6: a sixth of the widths of (1,2) (1,3) (1,4) (2,3) (2,4) (3,4)
    float2 *W6f = (float2 *)(smem + L.w6);  // the same as FP32 pairs (mixed path)
    C *A = (C *)(smem + L.A);
    C *B = (C *)(smem + L.B);
    R *F = (R *)(smem + L.F);
    const int tid = threadIdx.x, bd = blockDim.x;
    const MeshDev &m = a.mesh;
    const Fc4Dev &fc = a.fc;
    const R *mwm = mwm4_ptr<R>(fc);
    const C *egvs = egvs4_ptr<C>(P);
    const int64_t ld = (int64_t)m.n_full * N;
    const float sigfix32 = (float)P.sigma_fixed;
    C *T1 = reinterpret_cast<C *>(a.scratch) + (size_t)blockIdx.x * N3 * N;

    for (int t = blockIdx.x; t < a.n_quart; t += gridDim.x) {
        __syncthreads();  // the previous quartet's shared data is no longer read
        const QuartetRec rec = a.quart[t];
        const int qf[4] = {m.irr_full[rec.q1], rec.q2, rec.q3, rec.q4};
        const int qi[4] = {rec.q1, m.full_irr[rec.q2], m.full_irr[rec.q3], m.full_irr[rec.q4]};
        const uint32_t *mask = a.cand_mask + (size_t)rec.cand * 4;
        const int nred = rec.red_cnt;
        const int q2 = rec.q2, q3 = rec.q3, q4 = rec.q4;
        // permutation multiplicities (scattering_fourphonon.f90:104-122)
        double mult0, mult1;
        if (q2 == q3 && q3 == q4) {
            mult0 = 1.0;
            mult1 = 1.0;
        } else if ((q2 != q3 && q3 == q4) || (q3 != q2 && q2 == q4) || (q4 != q2 && q2 == q3)) {
            mult0 = 3.0;
            mult1 = 1.0;
        } else {
            mult0 = 6.0;
            mult1 = 2.0;
        }
        // ---- per-mode scalars, eigenvectors, equivalent quartets ----
        for (int i = tid; i < 4 * N; i += bd) {
            const int k = i / N, b = i % N;
            const size_t j = (size_t)qf[k] * N + b;
            const double w = P.omega[j];
            const float2 hl = P.omega_hl[j];  // NaN below 1e-9 Ha: no window holds it
            om[i] = w;
            sg[i] = P.sigsq[(size_t)qi[k] * N + b];
            be[i] = k > 0 ? P.be[(size_t)qi[k] * N + b] : 0.0;
            fo[i] = hl.x;
            fo[4 * N + i] = P.sigsq32[(size_t)qi[k] * N + b];
            fo[8 * N + i] = hl.y;
            if (k == 0) {
                inv1[b] = w > 0.0 ? 1.0 / w : 0.0;
                const int r = a.rows.rowidx[(size_t)rec.q1 * N + b];
                const bool on = (mask[b >> 5] >> (b & 31)) & 1u;
                rowid[b] = on ? r : -1;
                if (!on || r < 0) fo[b] = __int_as_float(0x7fc00000);
                wrow[b] = r >= 0 ? a.rows.weight4[r] : 0.0;
            }
        }
        for (int i = tid; i < nred && i < kMaxRed; i += bd) red[i] = a.red[rec.red_off + i];
        for (int i = tid; i < 4 * N2; i += bd) {
            const int k = i / N2, e = i % N2;
            const int r = e / N, b = e % N;
            E[i] = egvs[((size_t)qf[k] * N + b) * N + r];
        }
        if (it == 6)
            for (int i = tid; i < 6 * N2; i += bd) {
                const int which = i / N2, x = (i - which * N2) / N, y = i % N;
                const int k = which < 3 ? 0 : (which < 5 ? 1 : 2), l = which < 3 ? which + 1 : (which < 5 ? which - 1 : 3);
                const double w = adaptive_pair(P.vel + ((size_t)qf[k] * N + x) * 3, P.vel + ((size_t)qf[l] * N + y) * 3,
                                               P.reclat_g) / 6.0;
                if constexpr (DBL) W6d[i] = w;
                else W6f[i] = split_df(w);
            }
        if (tid == 0) *qlen = 0;
        __syncthreads();  // be[] of q2..q4 is in shared memory
        for (int i = tid; i < N2; i += bd) {
            const double n3 = be[2 * N + i / N], n4 = be[3 * N + i % N];
            P00[i] = (R)(n3 * n4);
            P11[i] = (R)((n3 + 1.0) * (n4 + 1.0));
        }
        for (int b = tid; b < N; b += bd) {
            const double n2 = be[N + b];
            N2v[b] = (R)n2;
            N2p[b] = (R)(n2 + 1.0);
            N2x3[b] = (R)(3.0 * n2);
            N2px3[b] = (R)(3.0 * (n2 + 1.0));
            N3v[b] = (R)be[2 * N + b];
            N4v[b] = (R)be[3 * N + b];
        }
        int g[3][3];
        {
            const int n12 = m.grid[1] * m.grid[2];
            for (int k = 0; k < 3; ++k) {
                const int q = qf[k + 1];
                g[k][0] = (q / n12) * m.lmul[0];  // g_d L/N_d
                g[k][1] = ((q / m.grid[2]) % m.grid[1]) * m.lmul[1];
                g[k][2] = (q % m.grid[2]) * m.lmul[2];
            }
        }
        // ---- ptf[a][bcd] (pretransform_phi4) into the T1 slice, one atom a1 at a time: the
        // force-constant quartets are sorted by atom block with a1 leading, so the phase
        // chunks of one a1 serve exactly its 3 n^3 outputs a = 3 a1 + i (n_fc4 * 81 real x
        // complex multiply-adds per q-quartet) ----
        constexpr int NA3 = NA * NA * NA;
        for (int a1 = 0; a1 < NA; ++a1) {
            C *ptf = T1 + (size_t)(3 * a1) * N3;
            const int t0 = fc.blk_ptr[a1 * NA3], t1 = fc.blk_ptr[(a1 + 1) * NA3];
            if (t0 >= t1) {
                for (int o = tid; o < 3 * N3; o += bd) ptf[o] = czero<C>();
                continue;
            }
            for (int c0 = t0; c0 < t1; c0 += phase_chunk4(N)) {
                const int cn = min(phase_chunk4(N), t1 - c0);
                __syncthreads();
                // K = sum_d ((g2 lv2 + g3 lv3 + g4 lv4)_d mod N_d) L/N_d mod L, evaluated as
                // (sum_d (g2 L/N_d) lv2 + ...) mod L: the same integer with one division
                for (int i = tid; i < cn; i += bd) {
                    const int32_t *lv = fc.lv + (size_t)(c0 + i) * 9;
                    int S = 0;
#pragma unroll
                    for (int d = 0; d < 3; ++d) S += g[0][d] * lv[d] + g[1][d] * lv[3 + d] + g[2][d] * lv[6 + d];
                    int K = S % m.L;
                    if (K < 0) K += m.L;
                    ph[i] = twiddle4<C>(a, K);
                }
                __syncthreads();
                for (int o = tid; o < 3 * N3; o += bd) {
                    const int i = o / N3, bcd = o % N3;
                    const int b = bcd / N2, c = (bcd / N) % N, d = bcd % N;
                    const int blk = ((a1 * NA + b / 3) * NA + c / 3) * NA + d / 3;
                    const int ijkl = i + (b % 3) * 3 + (c % 3) * 9 + (d % 3) * 27;
                    C acc = c0 == t0 ? czero<C>() : ptf[o];
                    const int lo = max(fc.blk_ptr[blk], c0), hi = min(fc.blk_ptr[blk + 1], c0 + cn);
                    for (int tt = lo; tt < hi; ++tt) {
                        const R mv = __ldg(mwm + (size_t)tt * 81 + ijkl);
                        const C p = ph[tt - c0];
                        acc.x = fma(mv, p.x, acc.x);
                        acc.y = fma(mv, p.y, acc.y);
                    }
                    ptf[o] = acc;
                }
            }
        }
        __syncthreads();
        // ---- T1[b1][bcd] = sum_a E1[a][b1] ptf[a][bcd], column by column in place (n^5
        // complex multiply-adds, against n_fc4 * 81 * n when E1 is folded into every
        // force-constant term) ----
        for (int col = tid; col < N3; col += bd) {
            C v[N];
#pragma unroll
            for (int x = 0; x < N; ++x) v[x] = T1[(size_t)x * N3 + col];
            for (int b1 = 0; b1 < N; ++b1) {
                if (rowid[b1] < 0) continue;
                C acc = czero<C>();
#pragma unroll
                for (int x = 0; x < N; ++x) cfma(acc, E[x * N + b1], v[x]);
                T1[(size_t)b1 * N3 + col] = acc;
            }
        }
        __syncthreads();
        const C *E2 = E + N2, *E3 = E + 2 * N2, *E4 = E + 3 * N2;
        for (int b0 = 0; b0 < N; b0 += NB) {
            if (NB == 1 && rowid[b0] < 0) continue;
            // ---- screen: a thread per (b1, b2, b3) of the batch; survivors queued (in no fixed
            // order: each writes its own F) ----
            for (int i = tid; i < NB * N2; i += bd) {
                const int b1 = b0 + i / N2, b23 = i % N2, b2 = b23 / N, b3 = b23 - b2 * N;
                const float f1 = fo[b1], f2 = fo[N + b2], f3 = fo[2 * N + b3];
                if (!(f1 == f1 && f2 == f2 && f3 == f3)) continue;
                const float s123 = fo[4 * N + b1] + fo[5 * N + b2] + fo[6 * N + b3];
                float w123 = 0.f;
                if (it == 6)
                    w123 = (float)P.thresh_sigma +
                           (DBL ? (float)(W6d[b1 * N + b2] + W6d[N2 + b1 * N + b3] + W6d[3 * N2 + b23])
                                : W6f[b1 * N + b2].x + W6f[N2 + b1 * N + b3].x + W6f[3 * N2 + b23].x);
                // om1 -+ om2 -+ om3, and the window's absolute margin
                const float pp = f1 - f2 - f3, mm = f1 + f2 + f3, pm = f1 - f2 + f3, mp = f1 + f2 - f3;
                for (int b4 = 0; b4 < N; ++b4) {
                    const float f4 = fo[3 * N + b4];
                    float s = sigfix32;
                    if (it == 2) s = sqrt_screen(s123 + fo[7 * N + b4]);
                    else if (it == 6)
                        s = w123 + (DBL ? (float)(W6d[2 * N2 + b1 * N + b4] + W6d[4 * N2 + b2 * N + b4] +
                                                  W6d[5 * N2 + b3 * N + b4])
                                        : W6f[2 * N2 + b1 * N + b4].x + W6f[4 * N2 + b2 * N + b4].x +
                                              W6f[5 * N2 + b3 * N + b4].x);
                    const float win = 8.0f * s * 1.001f + 1e-6f * (mm + f4);
                    const uint32_t live =
                        (fabsf(pp - f4) <= win ? 1u : 0u) | (mm + f4 <= win ? 2u : 0u) | (fabsf(mp - f4) <= win ? 4u : 0u) |
                        (fabsf(pm + f4) <= win ? 8u : 0u) | (fabsf(pm - f4) <= win ? 16u : 0u) |
                        (fabsf(mp + f4) <= win ? 32u : 0u) | (fabsf(pp + f4) <= win ? 64u : 0u) |
                        (fabsf(mm - f4) <= win ? 128u : 0u);
                    if (live) {
                        const unsigned on = __activemask();
                        const int lane = tid & 31, lead = __ffs(on) - 1;
                        int at = 0;
                        if (lane == lead) at = atomicAdd(qlen, __popc(on));
                        at = __shfl_sync(on, at, lead) + __popc(on & ((1u << lane) - 1u));
                        Q[at] = (uint32_t)(i * N + b4) | (live << 16);
                    }
                }
            }
            for (int i = tid; i < NB * N3; i += bd) F[i] = (R)0;
            // ---- second stage [b2][c][d] = sum_b E2[b][b2] T1[b1][b][c][d], third
            // [b2][b3][d] = sum_c E3[c][b3] [b2][c][d]; the fourth is the survivors' ----
            const C *T3;
            if constexpr (COLS) {
                for (int cd = tid; cd < N2; cd += bd) {
                    const C *t1 = T1 + (size_t)b0 * N3 + cd;
                    C acc[N];
#pragma unroll
                    for (int x = 0; x < N; ++x) acc[x] = czero<C>();
#pragma unroll 3
                    for (int b = 0; b < N; ++b) {
                        const C v = t1[b * N2];
#pragma unroll
                        for (int x = 0; x < N; ++x) cfma(acc[x], E2[b * N + x], v);
                    }
#pragma unroll
                    for (int x = 0; x < N; ++x) A[x * N2 + cd] = acc[x];
                }
                __syncthreads();
                for (int i = tid; i < N2; i += bd) {
                    const int b2 = i / N, d = i - b2 * N;
                    C *col = A + b2 * N2 + d;
                    C acc[N];
#pragma unroll
                    for (int x = 0; x < N; ++x) acc[x] = czero<C>();
#pragma unroll 3
                    for (int c = 0; c < N; ++c) {
                        const C v = col[c * N];
#pragma unroll
                        for (int x = 0; x < N; ++x) cfma(acc[x], E3[c * N + x], v);
                    }
#pragma unroll
                    for (int x = 0; x < N; ++x) col[x * N] = acc[x];
                }
                T3 = A;
            } else {
                for (int i = tid; i < NB * N3; i += bd) B[i] = T1[(size_t)b0 * N3 + i];
                __syncthreads();
                for (int i = tid; i < NB * N3; i += bd) {
                    const int b1 = i / N3, o = i - b1 * N3, b2 = o / N2, cd = o - b2 * N2;
                    C acc = czero<C>();
#pragma unroll
                    for (int b = 0; b < N; ++b) cfma(acc, E2[b * N + b2], B[b1 * N3 + b * N2 + cd]);
                    A[i] = acc;
                }
                __syncthreads();
                for (int i = tid; i < NB * N3; i += bd) {
                    const int k = i / N2, b3 = (i - k * N2) / N, d = i % N;  // k = (b1, b2)
                    C acc = czero<C>();
#pragma unroll
                    for (int c = 0; c < N; ++c) cfma(acc, E3[c * N + b3], A[k * N2 + c * N + d]);
                    B[i] = acc;
                }
                T3 = B;
            }
            __syncthreads();
            // ---- survivors: weights, Psi, F ----
            const int nq = *qlen;
            for (int s = tid; s < nq; s += bd) {
                const uint32_t qv = Q[s];
                const int o = (int)(qv & 0xffffu);
                uint32_t live = qv >> 16;
                const int b1 = b0 + o / N3, b2 = (o / N2) % N, b3 = (o / N) % N, b4 = o % N;
                R sigma, invsig, dd[4] = {(R)0, (R)0, (R)0, (R)0};
                if constexpr (DBL) {
                    if (it == 1) {
                        sigma = P.sigma_fixed;
                        invsig = 1.0 / sigma;
                    } else if (it == 2) {
                        const double sq = sg[b1] + sg[N + b2] + sg[2 * N + b3] + sg[3 * N + b4];
                        invsig = rsqrt(sq);
                        sigma = sq * invsig;
                    } else {
                        sigma = W6d[b1 * N + b2];
                        sigma += W6d[N2 + b1 * N + b3];
                        sigma += W6d[2 * N2 + b1 * N + b4];
                        sigma += W6d[3 * N2 + b2 * N + b3];
                        sigma += W6d[4 * N2 + b2 * N + b4];
                        sigma += W6d[5 * N2 + b3 * N + b4];
                        sigma += P.thresh_sigma;
                        invsig = 1.0 / sigma;
                    }
                } else {
                    if (it == 1) {
                        sigma = sigfix32;
                    } else if (it == 2) {
                        sigma = sqrtf(fo[4 * N + b1] + fo[5 * N + b2] + fo[6 * N + b3] + fo[7 * N + b4]);
                    } else {
                        float2 w = df_merge(W6f[b1 * N + b2], W6f[N2 + b1 * N + b3]);
                        w = df_merge(w, W6f[2 * N2 + b1 * N + b4]);
                        w = df_merge(w, W6f[3 * N2 + b2 * N + b3]);
                        w = df_merge(w, W6f[4 * N2 + b2 * N + b4]);
                        w = df_merge(w, W6f[5 * N2 + b3 * N + b4]);
                        sigma = w.x + (w.y + (float)P.thresh_sigma);
                    }
                    invsig = 1.0f / sigma;
                }
                const R win8 = (R)8 * sigma, h = (R)0.5 * invsig * invsig, cg = (R)kSqrt2PiInv * invsig;
                for (; live; live &= live - 1) {
                    const int j = __ffs(live) - 1;
                    const bool p2 = (kPlus2 >> j) & 1u, p3 = (kPlus3 >> j) & 1u, p4 = (kPlus4 >> j) & 1u;
                    R gj;
                    if constexpr (DBL) {
                        const double m2 = p2 ? om[N + b2] : -om[N + b2], m3 = p3 ? om[2 * N + b3] : -om[2 * N + b3],
                                     m4 = p4 ? om[3 * N + b4] : -om[3 * N + b4];
                        gj = gauss(om[b1] - (m2 + m3 + m4), win8, h, cg, P.exp2tab);
                    } else {
                        const float s2 = p2 ? 1.f : -1.f, s3 = p3 ? 1.f : -1.f, s4 = p4 ? 1.f : -1.f;
                        const float dx =
                            centre_diff4_f32(fo[b1], fo[8 * N + b1], s2 * fo[N + b2], s2 * fo[9 * N + b2], s3 * fo[2 * N + b3],
                                             s3 * fo[10 * N + b3], s4 * fo[3 * N + b4], s4 * fo[11 * N + b4]);
                        gj = fabsf(dx) > win8 ? 0.f : expf(-dx * dx * h) * cg;
                    }
                    const R sj = (j & 1) ? -gj : gj;
#pragma unroll
                    for (int k = 0; k < 4; ++k) dd[k] += (j >> 1) == k ? sj : (R)0;
                }
                if (dd[0] != (R)0 || dd[1] != (R)0 || dd[2] != (R)0 || dd[3] != (R)0) {
                    C psi = czero<C>();
                    const C *t3 = T3 + (o - b4);
#pragma unroll
                    for (int d = 0; d < N; ++d) cfma(psi, E4[d * N + b4], t3[d]);
                    const R ps = DBL ? psi.x * psi.x + psi.y * psi.y : fma(psi.x, psi.x, psi.y * psi.y);
                    // plf0 = (n2+1)(n3+1)(n4+1) - n2 n3 n4, plf1 = 3 n2 (n3+1)(n4+1) - (n2+1) n3 n4,
                    // plf2 = 3 n3 (n2+1)(n4+1) - (n3+1) n2 n4, plf3 = 3 n4 (n2+1)(n3+1) - (n4+1) n2 n3
                    const int k34 = b3 * N + b4;
                    const R n2 = N2v[b2], n2p = N2p[b2], p00 = P00[k34], p11 = P11[k34];
                    const R q1 = p00 + N3v[b3], q2x = p00 + N4v[b4];
                    const R acc = (R)mult0 * fma(n2p, p11, -n2 * p00) * dd[0];
                    R a1 = fma(N2x3[b2], p11, -n2p * p00) * dd[1];
                    a1 = fma(fma(N2px3[b2], q1, -n2 * q2x), dd[2], a1);
                    a1 = fma(fma(N2px3[b2], q2x, -n2 * q1), dd[3], a1);
                    const double w1 = wrow[b1];
                    F[o] = (R)(kFourPhononPrefactor * w1 * w1) * ps * fma((R)mult1, a1, acc);
                }
            }
            __syncthreads();
            // ---- sums over b4 (X) and over b3 (Y), in the queue's place, then R2, R3, R4, Gamma and
            // the row terms; the mixed path in double-float ----
            using Sum = typename std::conditional<DBL, double, float2>::type;
            Sum *X = (Sum *)Q, *Y = X + NB * N2;
            const auto clear = [](Sum &v) {
                if constexpr (DBL) v = 0.0;
                else v = make_float2(0.f, 0.f);
            };
            const auto add = [](Sum &v, R f) {
                if constexpr (DBL) v += f;
                else df_acc(v, f);
            };
            const auto merge = [](Sum &v, Sum w) {
                if constexpr (DBL) v += w;
                else v = df_merge(v, w);
            };
            if (tid == 0) *qlen = 0;
            for (int i = tid; i < 2 * NB * N2; i += bd) {
                const int e = i < NB * N2 ? i : i - NB * N2, k = e / N, x = e - k * N;  // k = (b1, b2); x = b3 or b4
                const R *f = i < NB * N2 ? F + e * N : F + k * N2 + x;
                const int step = i < NB * N2 ? 1 : N;
                Sum v;
                clear(v);
#pragma unroll
                for (int y = 0; y < N; ++y) add(v, f[y * step]);
                (i < NB * N2 ? X : Y)[e] = v;
            }
            __syncthreads();
            // R2[b2] = sum_b3 X, R3[b3] = sum_b2 X, R4[b4] = sum_b2 Y
            for (int i = tid; i < 3 * N * NB; i += bd) {
                const int b1 = i / (3 * N), e = i - b1 * 3 * N, which = e / N, b = e - which * N;
                const Sum *x = (which == 2 ? Y : X) + b1 * N2;
                Sum v;
                clear(v);
#pragma unroll
                for (int k = 0; k < N; ++k) merge(v, which == 0 ? x[b * N + k] : x[k * N + b]);
                double r;
                if constexpr (DBL) r = v;
                else r = (double)v.x + (double)v.y;
                if (which == 0) R2[b1 * N + b] = r;
                Rs[i] = nonzero(r) && rowid[b0 + b1] >= 0 ? 2.0 * r * om[(which + 1) * N + b] * inv1[b0 + b1] : 0.0;
            }
            __syncthreads();
            for (int b1 = tid; b1 < NB; b1 += bd) {
                const int row = rowid[b0 + b1];
                double gsum = 0.0;
                for (int b2 = 0; b2 < N; ++b2) gsum += R2[b1 * N + b2];
                if (row >= 0 && nonzero(gsum)) atomicAdd(a.gamma + row, (double)nred * gsum);
            }
            for (int i = tid; i < 3 * N * NB * nred; i += bd) {
                const int r = i / (3 * N * NB), k = i - r * 3 * N * NB, b1 = k / (3 * N), e = k - b1 * 3 * N;
                const int which = e / N, b = e - which * N, row = rowid[b0 + b1];
                const double v = Rs[k];
                if (!nonzero(v)) continue;
                const int4 pr = red[r];
                const int qp = which == 0 ? pr.x : (which == 1 ? pr.y : pr.z);
                atomicAdd(a.od + row * ld + (int64_t)qp * N + b, v);
            }
            // (the next batch's barriers separate its X and Rs from these reads; its queue does
            // not start before X is read: the barrier above)
        }
    }
}

template <int N, typename R>
int grid_n(int n_sm, int n_quart, bool it6) {
    const Layout4 L = make_layout4(N, sizeof(typename CT<R>::C), it6);
    const int per_sm = resident_ctas((const void *)k_fourphonon<N, R>, threads4_for(N), L.total, nullptr, nullptr);
    if (per_sm < 1) return 0;
    int grid = n_sm * per_sm;
    if (grid > n_quart) grid = n_quart;
    return grid < 1 ? 1 : grid;
}

template <int N, typename R>
cudaError_t launch_n4(const FourPhArgs &a, int grid, cudaStream_t s) {
    const Layout4 L = make_layout4(N, sizeof(typename CT<R>::C), a.ph.integrationtype == 6);
    k_fourphonon<N, R><<<grid, threads4_for(N), L.total, s>>>(a);
    return cudaGetLastError();
}

template <typename R>
int grid_prec(int n, int n_sm, int n_quart, bool it6) {
    switch (n) {
        case 3: return grid_n<3, R>(n_sm, n_quart, it6);
        case 6: return grid_n<6, R>(n_sm, n_quart, it6);
        case 9: return grid_n<9, R>(n_sm, n_quart, it6);
        case 12: return grid_n<12, R>(n_sm, n_quart, it6);
        case 15: return grid_n<15, R>(n_sm, n_quart, it6);
        default: return 0;
    }
}

template <typename R>
cudaError_t launch_prec4(const FourPhArgs &a, int grid, cudaStream_t s) {
    switch (a.mesh.n_mode) {
        case 3: return launch_n4<3, R>(a, grid, s);
        case 6: return launch_n4<6, R>(a, grid, s);
        case 9: return launch_n4<9, R>(a, grid, s);
        case 12: return launch_n4<12, R>(a, grid, s);
        case 15: return launch_n4<15, R>(a, grid, s);
        default: return cudaErrorNotSupported;
    }
}

}  // namespace

int fourphonon_grid(int n, int precision, int integrationtype, int n_sm, int n_quart) {
    const bool it6 = integrationtype == 6;
    if (n_quart <= 0) return 0;
    return precision == 0 ? grid_prec<double>(n, n_sm, n_quart, it6) : grid_prec<float>(n, n_sm, n_quart, it6);
}

size_t fourphonon_scratch_bytes(int n, int precision, int grid) {
    const size_t cs = precision == 0 ? sizeof(double2) : sizeof(float2);
    return (size_t)grid * n * n * n * n * cs;
}

cudaError_t launch_fourphonon(const FourPhArgs &a, int precision, int grid, cudaStream_t s) {
    if (a.n_quart <= 0 || grid <= 0) return cudaSuccess;
    if (precision == 0) return launch_prec4<double>(a, grid, s);
    return launch_prec4<float>(a, grid, s);
}

}  // namespace tdg
