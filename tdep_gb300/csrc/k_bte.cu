// The iterative BTE (kappa.f90:326-495): three kernels per iteration, the sums of F over the
// orbits (k_bte_sums), the products Xi F (k_bte_products) and the scalar recurrences with the
// foldout of the new F onto the full mesh (k_bte_update).
#include <cuda_runtime.h>

#include <algorithm>
#include <map>
#include <vector>

#include "dev_common.cuh"
#include "tdg_internal.cuh"

namespace tdg {

namespace {

// Two double-float accumulators (s, sl: high and low parts, one per column of a pair) +=
// x * f for the columns' elements (x, xl) and F values (f, fl); nx = -x. The scalar form per
// component: p = x f, pe = fma(x, f, -p), cross = fma(x, fl, xl f), TwoSum of s and p,
// sl += (e + pe) + cross. A subtraction a - b is fma(b, -1, a),
// rounded once as a - b is.
__device__ __forceinline__ void df2_fma(float2 &s, float2 &sl, float2 x, float2 nx, float2 xl, float2 f, float2 fl) {
    const float2 m1 = make_float2(-1.f, -1.f);
    const float2 p = __fmul2_rn(x, f);
    const float2 npe = __ffma2_rn(nx, f, p);  // p - x f = -pe exactly
    const float2 cross = __ffma2_rn(x, fl, __fmul2_rn(xl, f));
    const float2 t = __fadd2_rn(s, p);
    const float2 bb = __ffma2_rn(s, m1, t);                        // t - s
    const float2 e1 = __ffma2_rn(__ffma2_rn(bb, m1, t), m1, s);    // s - (t - bb)
    const float2 e = __fadd2_rn(e1, __ffma2_rn(bb, m1, p));       // + (p - bb)
    s = t;
    sl = __fadd2_rn(sl, __fadd2_rn(__ffma2_rn(npe, m1, e), cross));  // sl + ((e + pe) + cross)
}

// Three dot products per row of Xi (kappa.f90:411-413, the lo_gemv calls) over orbits.
// symmetrize_scatmat leaves the entries of a row equal on every orbit of the little group of
// its q1, so Xi F = sum over orbits and modes of Xi(orbit, b2) times the sum of F over the
// orbit's points: of Xi only the representatives' columns are kept (k_bte_compact), N/48 of
// N in all for a cubic crystal against the n_irr of the rows (0.52 of Xi at 16^3, 0.70 at
// 24^3). Points with the same little group have the same orbits: their rows are laid out
// together, and F is summed over the orbits once per group and iteration (k_bte_sums; some
// 20 groups at 24^3, 14 MB), not by every CTA of the products: that cost as much as the
// products, and 3 us of latency per chunk.
//   Format. GB300's FP64 pipe (2 FMA per SM and clock) would bound an FP64 product with
// three right-hand sides at ~1.2 TB/s of Xi, so it runs on the FP32 pipe: Xi and F as
// (hi, lo) float pairs with hi + lo = x to ~2^-48, each term accumulated in double-float
// (exact leading product by FMA, cross terms, TwoSum of the high parts); ~1e-14 relative,
// the bytes of FP64. Two neighbouring columns of a row are one float4 (hi of both, lo of
// both), so the arithmetic of the two runs in the packed FP32x2 instructions (__ffma2_rn,
// __fadd2_rn, __fmul2_rn: per component the scalar IEEE operation). Floats for Xi (half the
// bytes) fail the convergence test: the modes whose F is zero by symmetry (v = 0 at a
// high-symmetry point) carry 1e-7 of the typical |F| from the rounding of Xi, above the
// test's lo_sqtol floor, and rocksalt took 200 iterations, the limit, instead of 31-33.
//   Shape. The work is dealt out in equal parts to two CTAs per SM (bte_plan): a CTA has a few
// items, ranges of column pairs of up to kBteRows rows, and walks each in chunks of kBtePairs
// pairs. Its G x S warps take three rows and a share of the pairs each, Xi through a ring of
// kBteDepth steps that every lane fills for itself (cp.async, no barrier), the F sums from
// shared memory (two buffers, one barrier per chunk). The partial sums of an item stay in
// registers to its end and go to part[row][range][3] (FP64), added in range order by
// k_bte_update, so the result does not depend on scheduling.
//   Bound: HBM when Xi exceeds L2. Rocksalt 24^3: 1.15 GB in 217 us (5.3 TB/s, 0.79 of the
// measured copy rate) against 330 us for the whole of Xi, four or eight rows to a CTA;
// perovskite 16^3 96 us against 182; 40-atom supercell, no symmetry, 61 us against 72.
constexpr int kBteRows = 30;
constexpr int kBteThreads = 320;
constexpr int kBtePairs = 256;
constexpr int kBteDepth = 4;  // 10 warps x 4 steps x 1.5 KB and 24 KB of F sums: two CTAs per SM
constexpr size_t kBteSmem = sizeof(float4) * (2 * 3 * kBtePairs + kBteThreads * 3 * kBteDepth);

__device__ __forceinline__ void copy16(void *dst, const void *src, bool on) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(a), "l"(src), "r"(on ? 16 : 0) : "memory");
}

// Shares of the columns for G row groups of three: G S <= 10 warps, and kBteDepth steps of 32 S
// pairs divide a chunk.
__host__ __device__ constexpr int bte_share(int G) { return G <= 5 ? 2 : 1; }

__device__ __forceinline__ void products_item(const BteDev &d, const BteItem &it, const float4 *__restrict__ xi,
                                              float4 *smem) {
    const int n = d.n_mode, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int G = (it.n_row + 2) / 3, S = bte_share(G);
    const int g = w % G, s = w / G;
    float2 ah[3][3], al[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int x = 0; x < 3; ++x) ah[i][x] = al[i][x] = make_float2(0.f, 0.f);
    // F sums of the chunk from pair p on, with the thread's next group of copies
    auto fetch = [&](int p, float4 *buf) {
        for (int c = tid; c < 3 * kBtePairs; c += kBteThreads) {
            const int x = c / kBtePairs, pp = p + (c & (kBtePairs - 1));
            copy16(buf + c, d.fsum + it.fsum + (int64_t)x * it.n_pair + min(pp, it.n_pair - 1), pp < it.n_pair);
        }
    };
    // this warp's rows (the last one again past the item's); a lane's copies land in and are
    // read from its own places of the ring
    const float4 *xr[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) xr[i] = xi + it.xi + (int64_t)min(3 * g + i, it.n_row - 1) * it.n_pair;
    float4 *ring = smem + 2 * 3 * kBtePairs + w * (32 * 3 * kBteDepth) + lane;
    const bool work = s < S;
    int pc = it.p0 + s * 32 + lane;  // the pair to copy next
    auto copy = [&](int slot) {
        const bool on = work && pc < it.p1;
        const int at = min(pc, it.p1 - 1);
#pragma unroll
        for (int i = 0; i < 3; ++i) copy16(ring + (slot * 3 + i) * 32, xr[i] + at, on);
        asm volatile("cp.async.commit_group;" ::: "memory");
        pc += 32 * S;
    };
    fetch(it.p0, smem);
    asm volatile("cp.async.commit_group;" ::: "memory");
    for (int k = 0; k < kBteDepth - 1; ++k) copy(k);
    int cur = 0;
    for (int p = it.p0; p < it.p1; p += kBtePairs, cur ^= 1) {
        // the chunk's F sums are in the oldest group but the ring's last kBteDepth - 1 (a chunk
        // has at least kBteDepth steps; warps without rows have no ring)
        if (work)
            asm volatile("cp.async.wait_group %0;" ::"n"(kBteDepth - 1) : "memory");
        else
            asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();  // this chunk's sums are complete, the other buffer no longer read
        if (p + kBtePairs < it.p1) fetch(p + kBtePairs, smem + (cur ^ 1) * (3 * kBtePairs));
        if (work) {
            const float4 *fp = smem + cur * (3 * kBtePairs) + s * 32 + lane;
            for (int q = 0; q < kBtePairs && p + q < it.p1; q += 32 * kBteDepth * S) {
#pragma unroll
                for (int k = 0; k < kBteDepth; ++k) {
                    asm volatile("cp.async.wait_group %0;" ::"n"(kBteDepth - 2) : "memory");
                    float4 v[3];
#pragma unroll
                    for (int i = 0; i < 3; ++i) v[i] = ring[(k * 3 + i) * 32];
                    copy((k + kBteDepth - 1) % kBteDepth);
#pragma unroll
                    for (int x = 0; x < 3; ++x) {
                        const float4 f = fp[x * kBtePairs];
                        const float2 fh = make_float2(f.x, f.y), fl = make_float2(f.z, f.w);
#pragma unroll
                        for (int i = 0; i < 3; ++i)
                            df2_fma(ah[i][x], al[i][x], make_float2(v[i].x, v[i].y), make_float2(-v[i].x, -v[i].y),
                                    make_float2(v[i].z, v[i].w), fh, fl);
                    }
                    fp += 32 * S;
                }
            }
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    float2 *sh = reinterpret_cast<float2 *>(smem);  // [3 rows][S]
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            float2 a = df_merge(make_float2(ah[i][x].x, al[i][x].x), make_float2(ah[i][x].y, al[i][x].y));
            for (int o = 16; o > 0; o >>= 1) {
                float2 b;
                b.x = __shfl_xor_sync(0xffffffffu, a.x, o);
                b.y = __shfl_xor_sync(0xffffffffu, a.y, o);
                a = df_merge(a, b);
            }
            if (lane == 0 && s < S) sh[((3 * g + i) * 3 + x) * S + s] = a;
        }
    __syncthreads();
    if (tid < 3 * it.n_row) {
        float2 a = sh[tid * S];
        for (int k = 1; k < S; ++k) a = df_merge(a, sh[tid * S + k]);
        const int row = d.rows_by_group[it.row + tid / 3];
        d.part[((int64_t)row * d.split + it.range) * 3 + tid % 3] = (double)a.x + (double)a.y;
    }
}

__global__ void __launch_bounds__(kBteThreads, 2) k_bte_products(BteDev d, const BteItem *items, const int32_t *first,
                                                                 const float4 *__restrict__ xi) {
    extern __shared__ float4 smem[];  // F sums of a chunk's column pairs per direction, twice; the ring
    if (d.ctl->done) return;
    for (int k = first[blockIdx.x]; k < first[blockIdx.x + 1]; ++k) {
        __syncthreads();  // the previous item's sums are no longer read
        products_item(d, items[k], xi, smem);
    }
}

// The representatives' columns of Xi as double-float column pairs: pair p of a row holds
// columns 2p and 2p + 1 of its (orbit, mode) list as (hi, hi, lo, lo); an odd last column
// pairs with zero.
__global__ void k_bte_compact(int n, int64_t ld, int n_row, const BteRow *rows, const int32_t *rep, const double *xi,
                              float4 *out) {
    for (int r = blockIdx.y; r < n_row; r += gridDim.y) {
        const BteRow q = rows[r];
        const double *xr = xi + (int64_t)r * ld;
        float4 *o = out + q.xi;
        for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < q.n_pair; p += gridDim.x * blockDim.x) {
            float2 v[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int col = 2 * p + u, k = col / n;
                v[u] = col < q.n_col ? split_df(__ldcs(xr + (int64_t)rep[q.rep0 + k] * n + (col - k * n)))
                                     : make_float2(0.f, 0.f);
            }
            o[p] = make_float4(v[0].x, v[1].x, v[0].y, v[1].y);
        }
    }
}

// ---- the products over the non-zero elements alone ----
// Energy conservation empties most of a large mesh's Xi: a Gaussian reaches 8 sigma, and sigma
// shrinks with the mesh (rocksalt: 21 % of the elements are not zero at 12^3, 3.2 % at 24^3;
// perovskite 20 % at 16^3). Where few are left a row is the list of its non-zero elements, 12
// bytes each, and the F sums are gathered, 32 bytes per column from L2: rocksalt 24^3, 75
// iterations, call 22.9 -> 12.0 ms: an iteration takes 48 us where the dense products had
// alone taken 217; perovskite 16^3 102 us.
// A CTA takes an item of up to 2048 elements of a row, four gathers in flight per thread; the
// items' sums are added in order by k_bte_update.
__global__ void __launch_bounds__(256) k_bte_products_sparse(BteDev d) {
    __shared__ float2 sh[8][3];
    if (d.ctl->done) return;
    const BteSparseItem it = d.sparse[blockIdx.x];
    const float2 *val = d.sp_val + it.first;
    const int32_t *col = d.sp_col + it.first;
    const float4 *fs = d.fsum + it.fsum;
    const int tid = threadIdx.x;
    float2 a[3] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
    auto term = [](float2 &s, float2 v, float fh, float fl) {
        const float p = v.x * fh, pe = fmaf(v.x, fh, -p), cross = fmaf(v.x, fl, v.y * fh);
        const float t = s.x + p, bb = t - s.x;
        s.y += ((s.x - (t - bb)) + (p - bb)) + pe + cross;
        s.x = t;
    };
    for (int i0 = tid; i0 < it.count; i0 += 4 * 256) {
        float2 v[4];
        float4 f0[4];
        float2 f1[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int i = i0 + 256 * u;
            const bool on = i < it.count;
            v[u] = on ? __ldcs(val + i) : make_float2(0.f, 0.f);
            const float4 *f = fs + 2 * (int64_t)(on ? __ldcs(col + i) : 0);
            f0[u] = f[0];
            f1[u] = *reinterpret_cast<const float2 *>(f + 1);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (i0 + 256 * u >= it.count) break;
            term(a[0], v[u], f0[u].x, f0[u].y);
            term(a[1], v[u], f0[u].z, f0[u].w);
            term(a[2], v[u], f1[u].x, f1[u].y);
        }
    }
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        for (int o = 16; o > 0; o >>= 1)
            a[x] = df_merge(a[x], make_float2(__shfl_xor_sync(0xffffffffu, a[x].x, o),
                                              __shfl_xor_sync(0xffffffffu, a[x].y, o)));
        if ((tid & 31) == 0) sh[tid >> 5][x] = a[x];
    }
    __syncthreads();
    if (tid < 3) {
        float2 s = sh[0][tid];
        for (int w = 1; w < 8; ++w) s = df_merge(s, sh[w][tid]);
        d.part[(int64_t)blockIdx.x * 3 + tid] = (double)s.x + (double)s.y;
    }
}

// Element `col` of a row's (representative, mode) list.
__device__ __forceinline__ double bte_element(const double *xr, const int32_t *rep, const BteRow &q, int n, int col) {
    const int k = col / n;
    return __ldcs(xr + (int64_t)rep[q.rep0 + k] * n + (col - k * n));
}

// A CTA per row; four loads in flight per thread.
__global__ void __launch_bounds__(256) k_bte_count(int n, int64_t ld, int stride, const BteRow *rows, const int32_t *rep,
                                                   const double *xi, int32_t *nnz) {
    __shared__ int32_t total;
    const int r = blockIdx.x * stride;
    const BteRow q = rows[r];
    if (threadIdx.x == 0) total = 0;
    __syncthreads();
    int c = 0;
#pragma unroll 4
    for (int col = threadIdx.x; col < q.n_col; col += 256)
        c += bte_element(xi + (int64_t)r * ld, rep, q, n, col) != 0.0;
    c = __reduce_add_sync(0xffffffffu, c);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(&total, c);
    __syncthreads();
    if (threadIdx.x == 0) nnz[blockIdx.x] = total;
}

// A CTA per row, 1024 columns at a time: four consecutive blocks of 256, placed in column order.
__global__ void __launch_bounds__(256) k_bte_sparse(int n, int64_t ld, const BteRow *rows, const int32_t *rep,
                                                    const double *xi, const int64_t *first, float2 *val, int32_t *out) {
    __shared__ int cnt[2][4][8];
    const int r = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const BteRow q = rows[r];
    int64_t at = first[r];
    int buf = 0;
    for (int c0 = 0; c0 < q.n_col; c0 += 1024, buf ^= 1) {
        double v[4];
        uint32_t bal[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int col = c0 + 256 * u + (int)threadIdx.x;
            v[u] = col < q.n_col ? bte_element(xi + (int64_t)r * ld, rep, q, n, col) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            bal[u] = __ballot_sync(0xffffffffu, v[u] != 0.0);
            if (lane == 0) cnt[buf][u][w] = __popc(bal[u]);
        }
        __syncthreads();  // the other buffer's counts were read before it
        int total = 0;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            int before = 0, all = 0;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                before += j < w ? cnt[buf][u][j] : 0;
                all += cnt[buf][u][j];
            }
            if (v[u] != 0.0) {
                const int64_t k = at + total + before + __popc(bal[u] & ((1u << lane) - 1u));
                val[k] = split_df(v[u]);
                out[k] = c0 + 256 * u + (int)threadIdx.x;
            }
            total += all;
        }
        at += total;
    }
}

// Points of every orbit of the groups, one orbit after another: orbit i of group g starts at
// img_off[orb0 + i] (off: exclusive scan of the points per orbit over all q1; a q1's orbits
// cover the mesh once).
__global__ void k_bte_images(int n_full, int n_op, const BteGroup *grp, const int32_t *nuniq, const int32_t *img,
                             const int32_t *off, int32_t *img_off, int32_t *out) {
    const BteGroup g = grp[blockIdx.y];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.n_orb) return;
    const int k = g.rep0 + i;
    const int32_t *im = img + (size_t)k * n_op;
    const int at = off[k] - off[g.rep0] + (int)blockIdx.y * n_full;
    img_off[g.orb0 + i] = at;
    if (i == g.n_orb - 1) img_off[g.orb0 + i + 1] = at + nuniq[k];
    for (int u = 0; u < nuniq[k]; ++u) out[at + u] = im[u];
}

// F summed over the orbits of every group, as the products read it: [direction][column pair] of
// (hi, hi, lo, lo), or per column for the sparse form. `lanes` consecutive threads share a
// column's points (a sixth of the group's operations or so each: the chain of loads is what the
// kernel waits for).
__global__ void __launch_bounds__(256) k_bte_sums(BteDev d, const BteGroup *grp) {
    if (d.ctl->done) return;
    const BteGroup g = grp[blockIdx.y];
    const int n = d.n_mode, t = blockIdx.x * 256 + threadIdx.x;
    const int col = t / g.lanes, part = t - col * g.lanes, n_pair = (g.n_orb * n + 1) / 2;
    if ((blockIdx.x * 256) / g.lanes >= 2 * n_pair) return;
    float2 a[3] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
    if (col < g.n_orb * n) {
        const int o = col / n, b = col - o * n;
        const int i1 = d.img_off[g.orb0 + o + 1];
#pragma unroll 4
        for (int i = d.img_off[g.orb0 + o] + part; i < i1; i += g.lanes) {
            const float2 *f = d.fbb + (d.img[i] * n + b) * (int64_t)3;
#pragma unroll
            for (int x = 0; x < 3; ++x) a[x] = df_merge(a[x], f[x]);
        }
    }
    for (int o = 1; o < g.lanes; o <<= 1)
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            float2 v;
            v.x = __shfl_xor_sync(0xffffffffu, a[x].x, o);
            v.y = __shfl_xor_sync(0xffffffffu, a[x].y, o);
            a[x] = df_merge(a[x], v);
        }
    if (part != 0 || col >= 2 * n_pair) return;
    if (d.n_sparse) {  // [column] of (hi, lo) of the three directions, 32 bytes
        float4 *o = d.fsum + g.fsum / 3 * 4 + 2 * (int64_t)col;
        o[0] = make_float4(a[0].x, a[0].y, a[1].x, a[1].y);
        o[1] = make_float4(a[2].x, a[2].y, 0.f, 0.f);
        return;
    }
    float *out = reinterpret_cast<float *>(d.fsum + g.fsum + (col >> 1)) + (col & 1);
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        out[(int64_t)4 * x * n_pair] = a[x].x;
        out[(int64_t)4 * x * n_pair + 2] = a[x].y;
    }
}

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
            const double *p = d.part + (d.n_sparse ? (int64_t)d.part_first[r] : (int64_t)r * d.split) * 3 + x;
            for (int c = 0; c < d.ranges[r]; ++c) v += p[c * 3];
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

BtePlan bte_plan(int n, int n_irr, int n_sm, const int32_t *rep_ptr, const int32_t *row_count, int n_op,
                 const int32_t *irr_nop, const int32_t *irr_ops) {
    BtePlan pl;
    std::map<std::vector<int32_t>, int> ids;  // little group (its operations) -> group
    std::vector<std::vector<int32_t>> rows;   // rows of each group
    int row = 0;
    for (int q = 0; q < n_irr; ++q) {
        std::vector<int32_t> key(irr_ops + (size_t)q * n_op, irr_ops + (size_t)q * n_op + irr_nop[q]);
        std::sort(key.begin(), key.end());
        const auto at = ids.emplace(std::move(key), (int)pl.groups.size());
        if (at.second) {
            BteGroup g;
            g.rep0 = rep_ptr[q];
            g.n_orb = rep_ptr[q + 1] - rep_ptr[q];
            g.orb0 = pl.n_orb;
            g.fsum = pl.n_fsum;
            pl.n_fsum += 3 * (((int64_t)g.n_orb * n + 1) / 2);
            for (g.lanes = 1; g.lanes < 8 && 6 * g.lanes < irr_nop[q]; g.lanes *= 2) {}
            pl.sum_threads = std::max(pl.sum_threads, ((int64_t)g.n_orb * n + 1) * g.lanes);
            pl.n_orb += g.n_orb + 1;
            pl.max_orb = std::max(pl.max_orb, g.n_orb);
            pl.groups.push_back(g);
            rows.emplace_back();
        }
        for (int k = 0; k < row_count[q]; ++k) rows[at.first->second].push_back(row++);
    }
    // Equal shares of a group's rows, in multiples of three.
    auto share = [](int count) {
        const int k = (count + kBteRows - 1) / kBteRows;
        return ((count + k - 1) / k + 2) / 3 * 3;
    };
    // The row blocks one after another, each a number of units of columns (the steps between two
    // turns of the ring), cut into equal parts for two CTAs per SM: a CTA's fill and drain, some
    // 4 us, then come once or twice per iteration.
    const auto unit_of = [](int h) { return 32 * kBteDepth * bte_share((h + 2) / 3); };
    int64_t units = 0;
    for (size_t g = 0; g < rows.size(); ++g) {
        const int count = (int)rows[g].size();
        const int64_t pairs = ((int64_t)pl.groups[g].n_orb * n + 1) / 2;
        if (count == 0) continue;
        const int h = share(count);
        for (int k0 = 0; k0 < count; k0 += h) {
            const int u = unit_of(std::min(h, count - k0));
            units += (pairs + u - 1) / u;
        }
    }
    const int64_t parts = std::max<int64_t>(1, std::min<int64_t>(units, 2 * (int64_t)n_sm));
    int64_t done = 0;  // units dealt out
    pl.first.push_back(0);
    pl.rows.resize(row);
    pl.ranges.assign(row, 0);
    for (size_t g = 0; g < rows.size(); ++g) {
        const BteGroup &gr = pl.groups[g];
        const int count = (int)rows[g].size(), h = count ? share(count) : 3;
        const int32_t n_col = gr.n_orb * n, n_pair = (n_col + 1) / 2;
        for (int k0 = 0; k0 < count; k0 += h) {
            BteItem it;
            it.xi = pl.n_xi + (int64_t)k0 * n_pair;
            it.row = (int32_t)pl.by_group.size() + k0;
            it.n_row = std::min(h, count - k0);
            it.fsum = gr.fsum;
            it.n_pair = n_pair;
            it.range = 0;
            const int unit = unit_of(it.n_row);
            for (int64_t p = 0; p < n_pair; ++it.range) {
                // to the end of the part in hand or of the block
                const int64_t end = units * (int64_t)pl.first.size() / parts;
                const int64_t take = std::min<int64_t>(end - done, (n_pair - p + unit - 1) / unit);
                it.p0 = (int32_t)p;
                p = std::min<int64_t>(n_pair, p + take * unit);
                it.p1 = (int32_t)p;
                done += take;
                pl.items.push_back(it);
                if (done == end) pl.first.push_back((int32_t)pl.items.size());
            }
            for (int k = k0; k < k0 + it.n_row; ++k) pl.ranges[rows[g][k]] = it.range;
            pl.split = std::max(pl.split, it.range);
        }
        for (int k = 0; k < count; ++k) {
            BteRow &r = pl.rows[rows[g][k]];
            r.xi = pl.n_xi + (int64_t)k * n_pair;
            r.rep0 = gr.rep0;
            r.n_col = n_col;
            r.n_pair = n_pair;
        }
        pl.by_group.insert(pl.by_group.end(), rows[g].begin(), rows[g].end());
        pl.n_xi += (int64_t)count * n_pair;
    }
    return pl;
}

cudaError_t launch_bte_images(int n_full, int n_op, int n_group, int max_orb, const BteGroup *grp, const OrbitDev &o,
                              const int32_t *off, int32_t *img_off, int32_t *img, cudaStream_t s) {
    if (n_group <= 0 || max_orb <= 0) return cudaSuccess;
    dim3 grid((unsigned)((max_orb + 127) / 128), (unsigned)n_group);
    k_bte_images<<<grid, 128, 0, s>>>(n_full, n_op, grp, o.nuniq, o.img, off, img_off, img);
    return cudaGetLastError();
}

cudaError_t launch_bte_compact(int n, int64_t ld, int n_row, const BteRow *rows, const int32_t *rep, const double *xi,
                               float4 *out, cudaStream_t s) {
    if (n_row <= 0) return cudaSuccess;
    const int64_t bx = (ld / 2 + 255) / 256;
    dim3 grid((unsigned)std::max<int64_t>(1, std::min<int64_t>(bx, 64)), (unsigned)std::min(n_row, 65535));
    k_bte_compact<<<grid, 256, 0, s>>>(n, ld, n_row, rows, rep, xi, out);
    return cudaGetLastError();
}

cudaError_t launch_bte_count(int n, int64_t ld, int n_row, int stride, const BteRow *rows, const int32_t *rep,
                             const double *xi, int32_t *nnz, cudaStream_t s) {
    if (n_row <= 0) return cudaSuccess;
    k_bte_count<<<(n_row + stride - 1) / stride, 256, 0, s>>>(n, ld, stride, rows, rep, xi, nnz);
    return cudaGetLastError();
}

cudaError_t launch_bte_sparse(int n, int64_t ld, int n_row, const BteRow *rows, const int32_t *rep, const double *xi,
                              const int64_t *first, float2 *val, int32_t *col, cudaStream_t s) {
    if (n_row <= 0) return cudaSuccess;
    k_bte_sparse<<<n_row, 256, 0, s>>>(n, ld, rows, rep, xi, first, val, col);
    return cudaGetLastError();
}

cudaError_t launch_bte_products(const BteDev &d, const BteItem *items, const int32_t *first, int n_part, const float4 *xi,
                                cudaStream_t s) {
    if (d.n_sparse) {
        k_bte_products_sparse<<<d.n_sparse, 256, 0, s>>>(d);
        return cudaGetLastError();
    }
    if (n_part <= 0) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(k_bte_products, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBteSmem);
    if (e != cudaSuccess) return e;
    k_bte_products<<<n_part, kBteThreads, kBteSmem, s>>>(d, items, first, xi);
    return cudaGetLastError();
}

cudaError_t launch_bte_sums(const BteDev &d, const BteGroup *grp, int n_group, int64_t threads, cudaStream_t s) {
    if (n_group <= 0 || threads <= 0) return cudaSuccess;
    k_bte_sums<<<dim3((unsigned)((threads + 255) / 256), (unsigned)n_group), 256, 0, s>>>(d, grp);
    return cudaGetLastError();
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
