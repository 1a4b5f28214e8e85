// The iterative BTE (kappa.f90:326-495) around its products with Xi: one kernel per iteration
// for the scalar recurrences and the foldout of the new F onto the full mesh.
#include <cuda_runtime.h>

#include <vector>

#include "dev_common.cuh"
#include "tdg_internal.cuh"

namespace tdg {

namespace {

// foldout (kappa.f90:382-404): F of every point of the star of q1 from its irreducible point,
// Fbb(q, b) = sign(op) * R_|op| Fn(irr(q), b), one (point, mode) per thread and trip.
__device__ __forceinline__ void foldout_star(const BteDev &d, int q1, const double *fn) {
    const int n = d.n_mode;
    const int s0 = d.star_ptr[q1], total = (d.star_ptr[q1 + 1] - s0) * n;
    for (int i = threadIdx.x; i < total; i += blockDim.x) {
        const int iq = d.star[s0 + i / n], b = i % n;
        const int iop = d.full_op[iq];
        const double *m = d.op_cart + 9 * (abs(iop) - 1);
        const double *v = fn + b * 3;
        const double sg = iop > 0 ? 1.0 : -1.0;
        float2 *o = d.fbb + ((int64_t)iq * n + b) * 3;
        for (int x = 0; x < 3; ++x) o[x] = split_df(sg * (m[x] * v[0] + m[x + 3] * v[1] + m[x + 6] * v[2]));
    }
}

__global__ void k_bte_foldout(BteDev d) {
    foldout_star(d, blockIdx.x, d.fn + (size_t)blockIdx.x * d.n_mode * 3);
}

// One iteration after the products (kappa.f90:407-490), one CTA per irreducible point q1:
//   applyXi      Fnb = -(Xi F) / qs from the products' partial sums, added in range order;
//   distributeF  the degeneracy average in the reference's in-place order, then + F0: modes
//                whose degenerate sets do not meet do not affect each other, so every chain
//                of modes (bte_chains) and direction is one thread's, in ascending order;
//   addandcheck  relative change and mixing into Fn, a thread per mode;
//   foldout      of the new Fn onto the star of q1, for the next iteration's products.
// The CTA that finishes last adds the changes in order, tests convergence on the last three
// and advances the mixing. Returns at once when done is set (all CTAs of a kernel read it
// before the last one can set it).
// Bound: latency; a handful of dependent FP64 steps with a few hundred values. The same in
// five kernels with one thread per q1 for distributeF and addandcheck (whose divisions and
// table lookups then formed one chain) took 45 us an iteration at rocksalt 12^3 with its
// launches, 27 us of it that thread's.
__global__ void k_bte_update(BteDev d) {
    extern __shared__ double sm[];
    __shared__ double red[8];
    __shared__ int last;
    if (d.ctl->done) return;
    const int n = d.n_mode, m = 3 * n, tid = threadIdx.x, bd = blockDim.x, q1 = blockIdx.x;
    double *fb = sm, *f0 = sm + m, *fn = sm + 2 * m;
    const size_t base = (size_t)q1 * m;
    const double mixing = d.ctl->mixing;
    for (int i = tid; i < m; i += bd) {
        const int b1 = i / 3, x = i - 3 * b1;
        const int r = d.rowidx[q1 * n + b1];
        const double q = d.qs[q1 * n + b1];
        f0[i] = d.F0[base + i];
        fn[i] = d.fn[base + i];
        double v = 0.0;
        if (r >= 0 && !(q < kFreqTolD)) {
            const double *p = d.part + (int64_t)r * d.split * 3 + x;
            for (int c = 0; c < d.split; ++c) v += p[c * 3];
            v = -v / q;
        }
        fb[i] = v;
    }
    __syncthreads();
    for (int i = tid; i < m; i += bd) {
        const int b0 = i / 3, x = i - 3 * b0;
        int c = d.chain[q1 * n + b0];
        if (!(c & kChainFirst)) continue;
        for (int b = b0;;) {
            const int dg = d.degen[q1 * n + b];
            const int32_t *dm = d.degen_mode + ((size_t)q1 * n + b) * n;
            double v = 0.0;
            for (int j = 0; j < dg; ++j) v += fb[(dm[j] - 1) * 3 + x];
            if (dg != 1) v /= (double)dg;
            for (int j = 0; j < dg; ++j) fb[(dm[j] - 1) * 3 + x] = v;
            fb[b * 3 + x] = f0[b * 3 + x] + fb[b * 3 + x];
            b = (c & ~kChainFirst) - 1;
            if (b < 0) break;
            c = d.chain[q1 * n + b];
        }
    }
    __syncthreads();
    double g = 0.0;
    for (int b = tid; b < n; b += bd) {
        double g1 = 0.0, g2 = 0.0;
        for (int x = 0; x < 3; ++x) {
            const double v = fn[b * 3 + x], f = fb[b * 3 + x];
            g1 += (v - f) * (v - f);
            g2 += v * v;
            fn[b * 3 + x] = v * (1.0 - mixing) + mixing * f;
        }
        if (g2 > d.sqtol) g += g1 / g2;
    }
    for (int o = 16; o > 0; o >>= 1) g += __shfl_xor_sync(0xffffffffu, g, o);
    if ((tid & 31) == 0) red[tid >> 5] = g;
    __syncthreads();
    for (int i = tid; i < m; i += bd) d.fn[base + i] = fn[i];
    foldout_star(d, q1, fn);
    if (tid == 0) {
        double v = 0.0;
        for (int w = 0; w < (bd >> 5); ++w) v += red[w];
        d.change[q1] = v;
        __threadfence();
        last = atomicAdd(d.arrived, 1) == (int)gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    g = 0.0;
    for (int i = tid; i < (int)gridDim.x; i += bd) g += __ldcg(d.change + i);
    for (int o = 16; o > 0; o >>= 1) g += __shfl_xor_sync(0xffffffffu, g, o);
    if ((tid & 31) == 0) red[tid >> 5] = g;
    __syncthreads();
    if (tid != 0) return;
    g = 0.0;
    for (int w = 0; w < (bd >> 5); ++w) g += red[w];
    BteCtl *c = d.ctl;
    const int iter = c->iter + 1;
    d.scf[iter - 1] = g / d.n_irr / n;
    bool stop = false;
    if (iter >= 3) stop = d.scf[iter - 3] + d.scf[iter - 2] + d.scf[iter - 1] < d.tol;
    if (!stop && iter > 15 && mixing > 0.50) c->mixing = mixing * 0.98;
    c->iter = iter;
    *d.arrived = 0;
    if (stop || iter >= d.maxiter) c->done = 1;
}

}  // namespace

void bte_chains(int n_irr, int n_mode, const int32_t *degen, const int32_t *degen_mode, int32_t *chain) {
    std::vector<int> comp(n_mode), tail(n_mode);
    for (int q = 0; q < n_irr; ++q) {
        const int32_t *dg = degen + (size_t)q * n_mode, *dm = degen_mode + (size_t)q * n_mode * n_mode;
        int32_t *ch = chain + (size_t)q * n_mode;
        for (int b = 0; b < n_mode; ++b) comp[b] = b;
        for (int b = 0; b < n_mode; ++b)
            for (int j = 0; j < dg[b]; ++j) {
                const int to = comp[b], from = comp[dm[(size_t)b * n_mode + j] - 1];
                if (from != to)
                    for (int &x : comp)
                        if (x == from) x = to;
            }
        for (int b = 0; b < n_mode; ++b) tail[b] = -1;
        for (int b = 0; b < n_mode; ++b) {
            int &t = tail[comp[b]];
            ch[b] = t < 0 ? kChainFirst : 0;
            if (t >= 0) ch[t] += b + 1;
            t = b;
        }
    }
}

cudaError_t launch_bte_foldout(const BteDev &d, cudaStream_t s) {
    k_bte_foldout<<<d.n_irr, 128, 0, s>>>(d);
    return cudaGetLastError();
}

cudaError_t launch_bte_update(const BteDev &d, cudaStream_t s) {
    const size_t smem = sizeof(double) * 9 * (size_t)d.n_mode;
    k_bte_update<<<d.n_irr, d.n_mode > 42 ? 256 : 128, smem, s>>>(d);
    return cudaGetLastError();
}

}  // namespace tdg
