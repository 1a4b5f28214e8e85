// Isotope scattering and the two scattering-matrix symmetrisations.
#include <cuda_runtime.h>

#include <algorithm>

#include "dev_common.cuh"
#include "tdg_internal.cuh"

namespace tdg {

namespace {

constexpr double kIsotopePrefactor = 3.141592653589793 / 4.0;

__device__ __forceinline__ double block_sum(double v, double *sh) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) sh[w] = v;
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x == 0)
        for (int i = 0; i < (int)((blockDim.x + 31) / 32); ++i) s += sh[i];
    __syncthreads();
    return s;
}

// compute_isotope_scattering (scattering_isotope.f90:1-91). A CTA takes kIsoCols columns
// (q2, b2) of one row: an FP32 screen of the one Gaussian against its 8-sigma window (the
// margins of the three-phonon screen: a column it drops is exactly 0 in the reference), the
// survivors compacted into a queue, then the strength, width and Gaussian in FP64 by full
// warps. Bound: the FP64 pipe (2 lanes per clock and SM) for the survivors, a few per cent
// of the columns with adaptive widths. Forming the strength of every column first, with its
// 3 square roots per atom, cost 16.3 ms at perovskite 12^3 (32.6 M columns).
// |conj(u) v| = |u| |v|: the magnitudes are made once per mode and component
// (k_iso_mag), which leaves 3 products and 2 FMAs per atom.
constexpr int kIsoCols = 2048;

__global__ void k_iso_mag(int64_t ne, const double2 *egv, double *mag) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < ne) mag[i] = sqrt(egv[i].x * egv[i].x + egv[i].y * egv[i].y);
}

// Smearing width of -it 6 (scattering_isotope.f90:45-52): the velocity of (q2, b2) alone.
__device__ __forceinline__ double iso_width6(const PhononDev &ph, int64_t j) {
    const double *v = ph.vel + j * 3;
    double mx = 0.0;
    for (int jj = 0; jj < 3; ++jj) {
        double s = 0.0;
        for (int i = 0; i < 3; ++i) s += v[i] * ph.reclat_g[i + 3 * jj];
        mx = fmax(mx, s * s);
    }
    return sqrt(mx * 0.5) + ph.thresh_sigma;
}

// What the screen reads of a column: omega2 (NaN below 1e-9 Ha, which no window holds) and
// its share of the width (sigsq for -it 2, the width itself for -it 6).
__global__ void k_iso_cols(MeshDev m, PhononDev ph, float2 *col) {
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= (int64_t)m.n_full * m.n_mode) return;
    const int q2 = (int)(j / m.n_mode), b2 = (int)(j % m.n_mode);
    float w = 0.f;
    if (ph.integrationtype == 2) w = ph.sigsq32[(size_t)m.full_irr[q2] * m.n_mode + b2];
    if (ph.integrationtype == 6) w = (float)iso_width6(ph, j);
    col[j] = make_float2(ph.omega[j] < kFreqTolD ? __int_as_float(0x7fc00000) : ph.omega32[j], w);
}

__global__ void __launch_bounds__(256) k_isotope(MeshDev m, PhononDev ph, const int32_t *row_q1, const int32_t *row_b1,
                                                 const float2 *col, const double *mag, const double *disorder,
                                                 int32_t n_atom, double *gamma, double *xi) {
    constexpr int kPer = kIsoCols / 256;
    __shared__ double sh[32];
    __shared__ int wsum[33];
    __shared__ uint16_t queue[kIsoCols];
    const int n = m.n_mode, it = ph.integrationtype;
    const int r = blockIdx.y;
    const int q1 = row_q1[r], b1 = row_b1[r];
    const int f1 = m.irr_full[q1];
    const int64_t ld = (int64_t)m.n_full * n;
    const int64_t j0 = (int64_t)blockIdx.x * kIsoCols;
    const float fo1 = ph.omega32[(size_t)f1 * n + b1], fs1 = ph.sigsq32[(size_t)q1 * n + b1];
    const float sigfix = (float)ph.sigma_fixed;
    uint32_t live = 0u;
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
        const int64_t j = j0 + u * 256 + threadIdx.x;
        if (j >= ld) continue;
        const float2 c = __ldg(col + j);
        const float sg = it == 1 ? sigfix : (it == 2 ? sqrt_screen(fs1 + c.y) : c.y);
        if (fabsf(fo1 - c.x) <= 8.0f * sg * 1.001f + 1e-6f * (fo1 + c.x)) live |= 1u << u;
    }
    int nq = 0;
    int k = block_exclusive_scan(__popc(live), wsum, nq);
    for (; live; live &= live - 1) queue[k++] = (uint16_t)((__ffs(live) - 1) * 256 + threadIdx.x);
    __syncthreads();
    if (nq == 0) return;
    const double om1 = ph.omega[(size_t)f1 * n + b1], inv1 = ph.inv_omega[(size_t)f1 * n + b1];
    const double *e1 = mag + ((size_t)f1 * n + b1) * n;
    const double prefactor = kIsotopePrefactor * (1.0 / (double)m.n_full);
    double sum = 0.0;
    for (int i = threadIdx.x; i < nq; i += 256) {
        const int64_t j = j0 + queue[i];
        const double om2 = ph.omega[j];
        double sigma;
        if (it == 1) {
            sigma = ph.sigma_fixed;
        } else if (it == 2) {
            const int q2 = (int)(j / n), b2 = (int)(j - (int64_t)q2 * n);
            sigma = sqrt(ph.sigsq[(size_t)q1 * n + b1] + ph.sigsq[(size_t)m.full_irr[q2] * n + b2]);
        } else {
            sigma = iso_width6(ph, j);
        }
        if (fabs(om1 - om2) > 8.0 * sigma) continue;
        const double invsig = 1.0 / sigma;
        const double *e2 = mag + j * n;
        double strength = 0.0;
        for (int a = 0; a < n_atom; ++a) {
            const double fa = e1[3 * a] * e2[3 * a] + e1[3 * a + 1] * e2[3 * a + 1] + e1[3 * a + 2] * e2[3 * a + 2];
            strength = fma(fa * fa, disorder[a], strength);
        }
        const double dx = om1 - om2;
        const double gauss = exp_neg(dx * dx * 0.5 * invsig * invsig, ph.exp2tab) * kSqrt2PiInv * invsig;
        const double f0 = strength * prefactor * om1 * om2 * gauss;
        if (f0 != 0.0) xi[(int64_t)r * ld + j] += f0 * om2 * inv1;
        sum += f0;
    }
    const double s = block_sum(sum, sh);
    if (threadIdx.x == 0 && s != 0.0) atomicAdd(gamma + r, s);
}

// symmetrize_and_distribute (scattering_threephonon.f90:143-205, scattering_fourphonon.f90:195-250).
// Orbit tables of the little group of every irreducible q1, built once per mesh: q2 is a
// representative when no on-grid image is smaller (the reference's "cycle allq2" rule);
// its images are kept in operation order, -1 for operations that leave the grid.
__global__ void k_orbit_flag(MeshDev m, int32_t *flag) {
    const int q2 = blockIdx.x * blockDim.x + threadIdx.x;
    const int q1 = blockIdx.y;
    if (q2 >= m.n_full) return;
    const int nop = m.irr_nop[q1];
    const int32_t *ops = m.irr_ops + (size_t)q1 * m.n_op;
    int rep = 1;
    for (int j = 0; j < nop; ++j) {
        const int q2p = m.rot[(size_t)ops[j] * m.n_full + q2];
        if (q2p >= 0 && q2p < q2) {
            rep = 0;
            break;
        }
    }
    flag[(size_t)q1 * m.n_full + q2] = rep;
}

// Images are stored once each, in order of first appearance over the operations, with
// their multiplicity (operations that map q2 to the same point); cnt counts every
// on-grid operation, as the reference's averages do.
__global__ void k_orbit_fill(MeshDev m, const int32_t *flag, const int32_t *scan, OrbitDev o) {
    const int q2 = blockIdx.x * blockDim.x + threadIdx.x;
    const int q1 = blockIdx.y;
    if (q2 >= m.n_full) return;
    const size_t i = (size_t)q1 * m.n_full + q2;
    int32_t *orb_of = const_cast<int32_t *>(o.orb_of);
    if (!flag[i]) {
        orb_of[i] = -1;
        return;
    }
    const int k = scan[i];
    orb_of[i] = k;
    const_cast<int32_t *>(o.rep)[k] = q2;
    const int nop = m.irr_nop[q1];
    const int32_t *ops = m.irr_ops + (size_t)q1 * m.n_op;
    int32_t *img = const_cast<int32_t *>(o.img) + (size_t)k * m.n_op;
    int32_t *mult = const_cast<int32_t *>(o.mult) + (size_t)k * m.n_op;
    int c = 0, nu = 0;
    for (int j = 0; j < nop; ++j) {
        const int q2p = m.rot[(size_t)ops[j] * m.n_full + q2];
        if (q2p < 0) continue;
        ++c;
        int u = 0;
        while (u < nu && img[u] != q2p) ++u;
        if (u == nu) {
            img[nu] = q2p;
            mult[nu] = 0;
            ++nu;
        }
        ++mult[u];
    }
    const_cast<int32_t *>(o.cnt)[k] = c;
    const_cast<int32_t *>(o.nuniq)[k] = nu;
}

__device__ __forceinline__ bool positive(double v) { return __double_as_longlong(v) > 0; }  // v > 0, v not NaN

// symmetrize_and_distribute (scattering_threephonon.f90:143-205, scattering_fourphonon.f90:195-250)
// in place on one row per CTA: for every sampled q2 that represents its orbit, each mode's
// entries with od > 0 are averaged over the on-grid operations (images counted with their
// multiplicity) and the average is written to every image. Orbits are disjoint, so
// threads never touch the same entries; a bitmap ignores repeated entries of a sample
// (the reference would process them again to the same result).
// When xi != nullptr the symmetrised row is then added to xi.
__global__ void k_sym_distribute(MeshDev m, OrbitDev o, const int32_t *row_q1, const int64_t *rbeg,
                                 const int32_t *rlen, const int32_t *list, double *od, double *xi) {
    extern __shared__ uint32_t seen[];
    const int n = m.n_mode;
    const int r = blockIdx.x;
    const int q1 = row_q1[r];
    const int64_t ld = (int64_t)m.n_full * n;
    double *odr = od + (int64_t)r * ld;
    const int nw = (m.n_full + 31) / 32;
    for (int i = threadIdx.x; i < nw; i += blockDim.x) seen[i] = 0u;
    __syncthreads();
    for (int64_t qi = rbeg[r] + threadIdx.x; qi < rbeg[r] + rlen[r]; qi += blockDim.x) {
        const int q2 = list[qi] - 1;
        const int k = o.orb_of[(size_t)q1 * m.n_full + q2];
        if (k < 0) continue;
        const uint32_t bit = 1u << (q2 & 31);
        if (atomicOr(&seen[q2 >> 5], bit) & bit) continue;
        const int32_t *im = o.img + (size_t)k * m.n_op;
        const int32_t *mu = o.mult + (size_t)k * m.n_op;
        const int nu = o.nuniq[k];
        for (int b2 = 0; b2 < n; ++b2) {
            double buf = 0.0;
            int nn = 0;
            for (int u = 0; u < nu; ++u) {
                const double v = odr[(int64_t)im[u] * n + b2];
                if (positive(v)) {
                    nn += mu[u];
                    for (int rep = 0; rep < mu[u]; ++rep) buf += v;
                }
            }
            if (nn == 0) continue;
            const double avg = buf * o.rcp[nn];
            for (int u = 0; u < nu; ++u) odr[(int64_t)im[u] * n + b2] = avg;
        }
    }
    if (xi == nullptr) return;
    __syncthreads();
    double *xr = xi + (int64_t)r * ld;
    for (int64_t j = threadIdx.x; j < ld; j += blockDim.x) xr[j] += odr[j];
}

// Both row symmetrisations on tiles of whole orbits: symmetrize_and_distribute of the
// three-phonon terms (scattering_threephonon.f90:143-205; only orbits whose representative
// the row sampled, entries > 0 averaged) and symmetrize_scatmat (scattering.f90:296-357;
// every orbit, all entries). A CTA takes K = min(256, T / |G_q1|) consecutive orbits of its
// row's q1 (at most T points), gathers their images' n modes into shared memory with
// independent loads, averages there (each image weighted by its mult with one FMA, in
// first-appearance order: the reference adds it mult times, which differs in the last bit)
// and writes the images back; orbits that are +0 throughout are left alone (rocksalt 24^3, 97 %
// of the elements: call 12.0 -> 11.3 ms). With both passes in one kernel Xi crosses HBM once instead of
// twice. q1 whose little group is the identity
// alone are skipped: every orbit is one point with count 1, and both averages return it.
__global__ void __launch_bounds__(256) k_sym_tile(MeshDev m, OrbitDev o, const int32_t *row_q1, double *xi,
                                                  const uint32_t *sbits, int do_dist, int do_scat) {
    extern __shared__ double sym_sm[];
    __shared__ int wsum[8];
    const int n = m.n_mode, T = o.tile_pts;
    const int r = blockIdx.y, q1 = row_q1[r];
    const int nop = m.irr_nop[q1];
    if (nop <= 1) return;
    const int K = min(256, T / nop);
    const int kb = o.rep_ptr[q1], ke = o.rep_ptr[q1 + 1];
    const int k0 = kb + blockIdx.x * K;
    if (k0 >= ke) return;
    const int nk = min(K, ke - k0);
    double *vals = sym_sm;                                 // [T][n]
    double *pmud = vals + (size_t)T * n;                   // [T] multiplicity as a double
    int *pts = (int *)(pmud + T);                          // [T] image of each position
    int *pmu = pts + T;                                    // [T] its multiplicity
    int *off = pmu + T;                                    // [257] first position of each orbit
    const int tid = threadIdx.x;
    const int nu_t = tid < nk ? o.nuniq[k0 + tid] : 0;
    int P = 0;
    const int my = block_exclusive_scan(nu_t, wsum, P);
    if (tid < nk) {
        off[tid] = my;
        const int32_t *im = o.img + (size_t)(k0 + tid) * m.n_op;
        const int32_t *mu = o.mult + (size_t)(k0 + tid) * m.n_op;
        for (int u = 0; u < nu_t; ++u) {
            pts[my + u] = im[u];
            pmu[my + u] = mu[u];
            pmud[my + u] = (double)mu[u];  // converted once per image, not once per mode
        }
    }
    if (tid == 0) off[nk] = P;
    __syncthreads();
    double *xr = xi + (int64_t)r * m.n_full * n;
    // gather: eight independent loads in flight per thread before their stores (one load
    // per loop trip left each thread waiting on one gather at a time); p = e / n through
    // the float reciprocal, exact here (e < 2^13, and (e + 0.5) / n is at least 0.5 / n
    // from an integer)
    const int tot = P * n;
    const float inv_n = 1.0f / (float)n;
    constexpr int kGather = 8;
    for (int e0 = tid; e0 < tot; e0 += kGather * blockDim.x) {
        double v[kGather];
#pragma unroll
        for (int u = 0; u < kGather; ++u) {
            const int e = e0 + u * blockDim.x;
            const int p = (int)(((float)e + 0.5f) * inv_n), b2 = e - p * n;
            v[u] = e < tot ? xr[(int64_t)pts[p < P ? p : 0] * n + b2] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < kGather; ++u) {
            const int e = e0 + u * blockDim.x;
            if (e < tot) vals[e] = v[u];
        }
    }
    __syncthreads();
    const uint32_t *bits = sbits ? sbits + (size_t)r * ((m.n_full + 31) / 32) : nullptr;
    for (int it = tid; it < nk * n; it += blockDim.x) {
        const int t = it / n, b2 = it - t * n, k = k0 + t;
        const int p0 = off[t], p1 = off[t + 1];
        // Each image enters a sum once per operation that gives it: one FMA with its mult,
        // converted to double once per image (conversions run on the FP64 pipe too: the sums
        // are FP64 on a pipe of 2 operations per clock per SM, the bound of this kernel).
        // Most elements of a large mesh are +0 (no Gaussian reaches them): an orbit of such stays
        // as it is, without FP64 work and without being written back.
        long long any = 0;
        for (int p = p0; p < p1; ++p) any |= __double_as_longlong(vals[p * n + b2]);
        if (any == 0) continue;
        bool averaged = false;
        double avg = 0.0;
        if (do_dist) {
            const int q2 = o.rep[k];
            if ((bits[q2 >> 5] >> (q2 & 31)) & 1u) {
                double buf = 0.0;
                int nn = 0;
                for (int p = p0; p < p1; ++p) {
                    const double v = vals[p * n + b2];
                    if (__double_as_longlong(v) > 0) {  // v > 0, v not NaN
                        nn += pmu[p];
                        buf = fma(v, pmud[p], buf);
                    }
                }
                if (nn) {
                    avg = buf * o.rcp[nn];
                    averaged = true;
                }
            }
        }
        // symmetrize_scatmat: the mean over the operations, cnt = sum of mult; on an orbit the
        // distribution just set to one value that mean is the value itself
        if (do_scat && !averaged) {
            const int cnt = o.cnt[k];
            if (cnt) {
                double buf = 0.0;
                for (int p = p0; p < p1; ++p) buf = fma(vals[p * n + b2], pmud[p], buf);
                avg = buf * o.rcp[cnt];
                averaged = true;
            }
        }
        // a mean of exactly 0 (terms that cancel) is kept as -0: +0 is not written
        if (averaged)
            for (int p = p0; p < p1; ++p) vals[p * n + b2] = avg == 0.0 ? -0.0 : avg;
    }
    __syncthreads();
    for (int e = tid; e < tot; e += blockDim.x) {
        const double v = vals[e];
        if (__double_as_longlong(v) == 0) continue;
        const int p = (int)(((float)e + 0.5f) * inv_n), b2 = e - p * n;
        xr[(int64_t)pts[p] * n + b2] = v;
    }
}

// Bitmap of the q-points each row sampled, [n_row][ceil(n_full/32)] words, built in shared
// memory (dynamic, nw words) and written out once.
__global__ void k_sample_bits(int32_t n_full, const int64_t *rbeg, const int32_t *rlen, const int32_t *list,
                              uint32_t *bits) {
    extern __shared__ uint32_t sb[];
    const int r = blockIdx.x, nw = (n_full + 31) / 32;
    for (int i = threadIdx.x; i < nw; i += blockDim.x) sb[i] = 0u;
    __syncthreads();
    for (int64_t i = rbeg[r] + threadIdx.x; i < rbeg[r] + rlen[r]; i += blockDim.x) {
        const int q2 = list[i] - 1;
        atomicOr(sb + (q2 >> 5), 1u << (q2 & 31));
    }
    __syncthreads();
    uint32_t *br = bits + (size_t)r * nw;
    for (int i = threadIdx.x; i < nw; i += blockDim.x) br[i] = sb[i];
}

}  // namespace

cudaError_t launch_iso_mag(int64_t ne, const double2 *egv, double *mag, cudaStream_t s) {
    if (ne <= 0) return cudaSuccess;
    k_iso_mag<<<(unsigned)((ne + 255) / 256), 256, 0, s>>>(ne, egv, mag);
    return cudaGetLastError();
}

cudaError_t launch_isotope(const MeshDev &m, const PhononDev &ph, const RowsDev &rows, const int32_t *row_q1,
                           const int32_t *row_b1, float2 *col, const double *mag, const double *disorder,
                           int32_t n_atom, double *gamma, double *xi, cudaStream_t s) {
    if (rows.n_row <= 0) return cudaSuccess;
    const int64_t ld = (int64_t)m.n_full * m.n_mode;
    k_iso_cols<<<(unsigned)((ld + 255) / 256), 256, 0, s>>>(m, ph, col);
    dim3 grid((unsigned)((ld + kIsoCols - 1) / kIsoCols), (unsigned)rows.n_row);
    k_isotope<<<grid, 256, 0, s>>>(m, ph, row_q1, row_b1, col, mag, disorder, n_atom, gamma, xi);
    return cudaGetLastError();
}

namespace {
__global__ void k_rep_ptr(const int32_t *scan, int32_t n_irr, int32_t n_full, int32_t *rep_ptr) {
    const int q1 = blockIdx.x * blockDim.x + threadIdx.x;
    if (q1 <= n_irr) rep_ptr[q1] = scan[(size_t)q1 * n_full];
}
}  // namespace

cudaError_t launch_orbit_flag(const MeshDev &m, int32_t *flag, cudaStream_t s) {
    dim3 grid((unsigned)((m.n_full + 127) / 128), (unsigned)m.n_irr);
    k_orbit_flag<<<grid, 128, 0, s>>>(m, flag);
    return cudaGetLastError();
}

cudaError_t launch_orbit_fill(const MeshDev &m, const int32_t *flag, const int32_t *scan, OrbitDev &o,
                              cudaStream_t s) {
    dim3 grid((unsigned)((m.n_full + 127) / 128), (unsigned)m.n_irr);
    k_orbit_fill<<<grid, 128, 0, s>>>(m, flag, scan, o);
    k_rep_ptr<<<(m.n_irr + 1 + 127) / 128, 128, 0, s>>>(scan, m.n_irr, m.n_full, const_cast<int32_t *>(o.rep_ptr));
    return cudaGetLastError();
}

cudaError_t launch_sym_distribute(const MeshDev &m, const OrbitDev &o, int32_t n_row, const int32_t *row_q1,
                                  const int64_t *rbeg, const int32_t *rlen, const int32_t *list, double *od, double *xi,
                                  cudaStream_t s) {
    if (n_row <= 0) return cudaSuccess;
    const size_t sm = sizeof(uint32_t) * (size_t)((m.n_full + 31) / 32);
    if (sm > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(k_sym_distribute, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
        if (e != cudaSuccess) return e;
    }
    k_sym_distribute<<<n_row, 256, sm, s>>>(m, o, row_q1, rbeg, rlen, list, od, xi);
    return cudaGetLastError();
}

int sym_tile_points(int n_mode) {
    const int t = 4096 / (n_mode > 0 ? n_mode : 1);
    return t < 64 ? 64 : (t > 1024 ? 1024 : t);
}

size_t sym_tile_smem(int n_mode) {
    const int T = sym_tile_points(n_mode);
    return sizeof(double) * (size_t)T * (n_mode + 1) + sizeof(int) * (2 * (size_t)T + 257);
}

int sym_tile_count(int n_rep, int n_ops, int n_mode) {
    if (n_ops <= 1 || n_rep <= 0) return 0;
    int K = sym_tile_points(n_mode) / n_ops;
    K = K > 256 ? 256 : K;
    return (n_rep + K - 1) / K;
}

cudaError_t launch_sample_bits(int32_t n_full, int32_t n_row, const int64_t *rbeg, const int32_t *rlen,
                               const int32_t *list, uint32_t *bits, cudaStream_t s) {
    if (n_row <= 0) return cudaSuccess;
    const size_t sm = sizeof(uint32_t) * (size_t)((n_full + 31) / 32);
    if (sm > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(k_sample_bits, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
        if (e != cudaSuccess) return e;
    }
    k_sample_bits<<<n_row, 256, sm, s>>>(n_full, rbeg, rlen, list, bits);
    return cudaGetLastError();
}

cudaError_t launch_sym_tile(const MeshDev &m, const OrbitDev &o, int32_t n_row, const int32_t *row_q1, double *xi,
                            const uint32_t *sbits, bool dist, bool scat, cudaStream_t s) {
    if (n_row <= 0 || o.max_tiles <= 0 || (!dist && !scat)) return cudaSuccess;
    const size_t sm = sym_tile_smem(m.n_mode);
    if (sm > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(k_sym_tile, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
        if (e != cudaSuccess) return e;
    }
    dim3 grid((unsigned)o.max_tiles, (unsigned)n_row);
    k_sym_tile<<<grid, 256, sm, s>>>(m, o, row_q1, xi, sbits, dist ? 1 : 0, scat ? 1 : 0);
    return cudaGetLastError();
}

namespace {
// rot[o][q] = full-mesh index of R_o q, -1 when R_o q is off the mesh: (R q)_i = num / L with
// num = sum_j R_ij g_j (L / N_j) in 32-bit integers (|num| < 3 L max N), on the mesh when
// num is a multiple of L / N_i.
__global__ void k_rot_table(int g0, int g1, int g2, int L, int n_full, const int32_t *op_recfrac, int32_t *rot) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    const int o = blockIdx.y;
    if (q >= n_full) return;
    const int32_t *R = op_recfrac + 9 * o;
    const int g[3] = {g0, g1, g2};
    const int gi[3] = {q / (g1 * g2), (q / g2) % g1, q % g2};
    int out[3];
    for (int i = 0; i < 3; ++i) {
        const int num = R[i] * gi[0] * (L / g0) + R[i + 3] * gi[1] * (L / g1) + R[i + 6] * gi[2] * (L / g2);
        const int step = L / g[i];
        if (num % step != 0) {
            rot[(size_t)o * n_full + q] = -1;
            return;
        }
        int v = (num / step) % g[i];
        if (v < 0) v += g[i];
        out[i] = v;
    }
    rot[(size_t)o * n_full + q] = (out[0] * g1 + out[1]) * g2 + out[2];
}

// Eigenvectors scaled by 1/sqrt(omega) (scattering_threephonon.f90:67,93,102), FP64 and FP32,
// zero for omega < lo_freqtol; IEEE sqrt and division as on the host.
__global__ void k_egv_scaled(int64_t nm, int n, const double2 *egv, const double *omega, double2 *egvs,
                             float2 *egvs32) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nm * n) return;
    const double om = omega[i / n];
    double2 v = make_double2(0.0, 0.0);
    if (!(om < kFreqTolD)) {
        const double sq = sqrt(om);
        const double2 e = egv[i];
        v = make_double2(e.x / sq, e.y / sq);
    }
    egvs[i] = v;
    egvs32[i] = make_float2((float)v.x, (float)v.y);
}
}  // namespace

cudaError_t launch_rot_table(const int32_t grid[3], int L, int n_full, int n_op, const int32_t *op_recfrac,
                             int32_t *rot, cudaStream_t s) {
    if (n_full <= 0 || n_op <= 0) return cudaSuccess;
    dim3 g((unsigned)((n_full + 255) / 256), (unsigned)n_op);
    k_rot_table<<<g, 256, 0, s>>>(grid[0], grid[1], grid[2], L, n_full, op_recfrac, rot);
    return cudaGetLastError();
}

cudaError_t launch_egv_scaled(int64_t nm, int n, const double2 *egv, const double *omega, double2 *egvs,
                              float2 *egvs32, cudaStream_t s) {
    const int64_t total = nm * n;
    if (total <= 0) return cudaSuccess;
    k_egv_scaled<<<(unsigned)((total + 255) / 256), 256, 0, s>>>(nm, n, egv, omega, egvs, egvs32);
    return cudaGetLastError();
}

}  // namespace tdg
