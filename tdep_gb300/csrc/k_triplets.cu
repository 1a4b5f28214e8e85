// K1: irreducible q-triplet and q-quartet enumeration on integer rotation tables.
//
// For every candidate (q1 irreducible, q2 from the Monte-Carlo sample of q1's rows):
//   q3 = -q1-q2 mod G                          (lo_fftgrid_helper.f90:136-163)
//   skip q3 < q2                               (scattering_threephonon.f90:75)
//   triplet_is_irreducible                     (scattering_threephonon.f90:319-448)
// The reference rotates fractional coordinates in floating point and rounds back to the
// grid; here every rotated index comes from a host-built table rot[op][q], so the whole
// enumeration is integer arithmetic and bit-exact.
// Two passes: count (accepted flag and number of equivalent triplets per candidate),
// exclusive scan, fill. Output order equals candidate order, so results are deterministic.
#include "tdg_internal.cuh"

namespace tdg {

namespace {

constexpr int kMaxOps = 192;

__device__ __forceinline__ void grid_coords(const MeshDev &m, int q, int &i, int &j, int &k) {
    const int n12 = m.grid[1] * m.grid[2];
    i = q / n12;
    j = (q / m.grid[2]) % m.grid[1];
    k = q % m.grid[2];
}

__device__ __forceinline__ int wrap(int x, int n) {
    x %= n;
    return x < 0 ? x + n : x;
}

// q3 = -q1-q2 (0-based full indices).
__device__ __forceinline__ int third_index(const MeshDev &m, int f1, int q2) {
    int i1, j1, k1, i2, j2, k2;
    grid_coords(m, f1, i1, j1, k1);
    grid_coords(m, q2, i2, j2, k2);
    const int i3 = wrap(-i1 - i2, m.grid[0]);
    const int j3 = wrap(-j1 - j2, m.grid[1]);
    const int k3 = wrap(-k1 - k2, m.grid[2]);
    return (i3 * m.grid[1] + j3) * m.grid[2] + k3;
}

// q4 = -q1-q2-q3.
__device__ __forceinline__ int fourth_index(const MeshDev &m, int f1, int q2, int q3) {
    int i1, j1, k1, i2, j2, k2, i3, j3, k3;
    grid_coords(m, f1, i1, j1, k1);
    grid_coords(m, q2, i2, j2, k2);
    grid_coords(m, q3, i3, j3, k3);
    const int i4 = wrap(-i1 - i2 - i3, m.grid[0]);
    const int j4 = wrap(-j1 - j2 - j3, m.grid[1]);
    const int k4 = wrap(-k1 - k2 - k3, m.grid[2]);
    return (i4 * m.grid[1] + j4) * m.grid[2] + k4;
}

// Images (x, y) of (q2, q3) under operation j of q1's little group; false where one of them
// is off the mesh.
__device__ __forceinline__ bool triplet_image(const MeshDev &m, const int32_t *ops, int j, int q2, int q3, int &x,
                                              int &y) {
    const int32_t *rot = m.rot + (size_t)ops[j] * m.n_full;
    x = rot[q2];
    y = rot[q3];
    return x >= 0 && y >= 0;
}

// triplet_is_irreducible's first test: no image has its smaller point above q2.
__device__ __forceinline__ bool triplet_accepted(const MeshDev &m, int q1, int q2, int q3) {
    const int nop = m.irr_nop[q1];
    const int32_t *ops = m.irr_ops + (size_t)q1 * m.n_op;
    for (int j = 0; j < nop; ++j) {
        int x, y;
        if (triplet_image(m, ops, j, q2, q3, x, y) && min(x, y) > q2) return false;
    }
    return true;
}

// The distinct equivalent triplets of an accepted one: an operation counts unless a later one
// gives the same pair (in either order); operations off the mesh give (q2, q3). Returns their
// number; when out != nullptr they are written in operation order (unsorted pairs).
// Up to kLaneOps operations one thread compares all pairs of them (triplet_images); larger
// little groups take a warp, 32 operations at a time (triplet_images_warp): at the zone
// centre of a cubic mesh one thread with 48 operations in local memory held the kernel for
// 50 us whatever the mesh.
constexpr int kLaneOps = 4;

__device__ __forceinline__ int triplet_images(const MeshDev &m, int q1, int q2, int q3, int2 *out) {
    const int nop = m.irr_nop[q1];
    const int32_t *ops = m.irr_ops + (size_t)q1 * m.n_op;
    int x[kLaneOps], y[kLaneOps], cnt = 0;
#pragma unroll
    for (int j = 0; j < kLaneOps; ++j)
        if (j >= nop || !triplet_image(m, ops, j, q2, q3, x[j], y[j])) {
            x[j] = q2;
            y[j] = q3;
        }
#pragma unroll
    for (int j = 0; j < kLaneOps; ++j) {
        bool uniq = j < nop;
#pragma unroll
        for (int k = j + 1; k < kLaneOps; ++k)
            if (k < nop && ((x[k] == x[j] && y[k] == y[j]) || (x[k] == y[j] && y[k] == x[j]))) uniq = false;
        if (uniq) {
            if (out) out[cnt] = make_int2(x[j], y[j]);
            ++cnt;
        }
    }
    return cnt;
}

// All lanes of a full warp with the same arguments.
__device__ int triplet_images_warp(const MeshDev &m, int q1, int q2, int q3, int2 *out) {
    constexpr int kChunks = kMaxOps / 32;
    const int nop = m.irr_nop[q1], lane = threadIdx.x & 31, nch = (nop + 31) / 32;
    const int32_t *ops = m.irr_ops + (size_t)q1 * m.n_op;
    unsigned long long key[kChunks];
    int2 img[kChunks];
#pragma unroll
    for (int c = 0; c < kChunks; ++c) {
        const int j = c * 32 + lane;
        int x = q2, y = q3;
        if (j < nop && !triplet_image(m, ops, j, q2, q3, x, y)) {
            x = q2;
            y = q3;
        }
        img[c] = make_int2(x, y);
        // no pair has this key: lanes past the last operation match one another only
        key[c] = j < nop ? ((unsigned long long)(unsigned)min(x, y) << 32) | (unsigned)max(x, y) : ~0ULL;
    }
    int cnt = 0;
#pragma unroll
    for (int c = 0; c < kChunks; ++c) {
        if (c >= nch) break;
        const unsigned same = __match_any_sync(0xffffffffu, key[c]);
        bool uniq = c * 32 + lane < nop && (same >> lane) == 1u;  // the last of them in this chunk
#pragma unroll
        for (int d = c + 1; d < kChunks; ++d) {
            if (d >= nch) break;
            const int left = min(32, nop - d * 32);
            for (int l = 0; l < left; ++l)
                if (__shfl_sync(0xffffffffu, key[d], l) == key[c]) uniq = false;
        }
        const unsigned in = __ballot_sync(0xffffffffu, uniq);
        if (out && uniq) out[cnt + __popc(in & ((1u << lane) - 1u))] = img[c];
        cnt += __popc(in);
    }
    return cnt;
}

__device__ __forceinline__ void sort3(int &x, int &y, int &z) {
    if (x > y) { int t = x; x = y; y = t; }
    if (y > z) { int t = y; y = z; z = t; }
    if (x > y) { int t = x; x = y; y = t; }
}

// quartet_is_irreducible (scattering_fourphonon.f90:330-456). Off-grid operations keep
// their original (unsorted) triple replaced by (q2,q3,q4) while their sorted copy stays
// at the sentinel, exactly as the reference's two successive replacement tests do.
__device__ int quartet_images(const MeshDev &m, int q1, int q2, int q3, int q4, int4 *out) {
    const int nop = m.irr_nop[q1];
    const int32_t *ops = m.irr_ops + (size_t)q1 * m.n_op;
    int a[kMaxOps], b[kMaxOps], c[kMaxOps];
    bool isred = false;
    constexpr int kSentinel = -2147483647;
    for (int j = 0; j < nop; ++j) {
        const int o = ops[j];
        const int x = m.rot[(size_t)o * m.n_full + q2];
        const int y = m.rot[(size_t)o * m.n_full + q3];
        const int z = m.rot[(size_t)o * m.n_full + q4];
        if (x < 0 || y < 0 || z < 0) {
            a[j] = kSentinel;
            b[j] = kSentinel;
            c[j] = kSentinel;
            continue;
        }
        a[j] = x;
        b[j] = y;
        c[j] = z;
        int s0 = x, s1 = y, s2 = z;
        sort3(s0, s1, s2);
        if (s0 > q2 || s1 > q3) isred = true;
    }
    if (isred) return -1;
    int cnt = 0;
    for (int j = 0; j < nop; ++j) {
        int s0 = a[j], s1 = b[j], s2 = c[j];
        if (a[j] != kSentinel) sort3(s0, s1, s2);
        bool uniq = true;
        for (int k = j + 1; k < nop; ++k) {
            int t0 = a[k], t1 = b[k], t2 = c[k];
            if (a[k] != kSentinel) sort3(t0, t1, t2);
            if (t0 == s0 && t1 == s1 && t2 == s2) {
                uniq = false;
                break;
            }
        }
        if (uniq) {
            if (out) {
                if (a[j] == kSentinel)
                    out[cnt] = make_int4(q2, q3, q4, 0);
                else
                    out[cnt] = make_int4(a[j], b[j], c[j], 0);
            }
            ++cnt;
        }
    }
    return cnt;
}

__global__ void k_triplet_count(MeshDev m, const int4 *cand, int32_t n_cand, int32_t *n_trip, int32_t *n_red,
                                int32_t *status) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
    int q1 = 0, q2 = 0, q3 = 0, nr = 0;
    bool on = false, warp = false;
    if (c < n_cand) {
        q1 = cand[c].x;
        q2 = cand[c].y;
        if (q1 < 0 || q1 >= m.n_irr || q2 < 0 || q2 >= m.n_full || m.irr_nop[q1] > kMaxOps) {
            atomicCAS(status, kDevOk, kDevBadIndex);
        } else {
            q3 = third_index(m, m.irr_full[q1], q2);
            on = q3 >= q2 && triplet_accepted(m, q1, q2, q3);
            warp = on && m.irr_nop[q1] > kLaneOps;
            if (on && !warp) nr = triplet_images(m, q1, q2, q3, nullptr);
        }
    }
    for (unsigned left = __ballot_sync(0xffffffffu, warp); left; left &= left - 1) {
        const int l = __ffs(left) - 1;
        const int k = triplet_images_warp(m, __shfl_sync(0xffffffffu, q1, l), __shfl_sync(0xffffffffu, q2, l),
                                          __shfl_sync(0xffffffffu, q3, l), nullptr);
        if (lane == l) nr = k;
    }
    if (c >= n_cand) return;
    n_trip[c] = on ? 1 : 0;
    n_red[c] = nr;
}

__global__ void k_triplet_fill(MeshDev m, const int4 *cand, int32_t n_cand, const int32_t *trip_off,
                               const int32_t *red_off, TripletRec *trip, int2 *red) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    int q1 = 0, q2 = 0, q3 = 0, at = 0;
    bool warp = false;
    if (c < n_cand && trip_off[c + 1] != trip_off[c]) {
        q1 = cand[c].x;
        q2 = cand[c].y;
        q3 = third_index(m, m.irr_full[q1], q2);
        at = red_off[c];
        TripletRec r;
        r.q1 = q1;
        r.q2 = q2;
        r.q3 = q3;
        r.cand = cand[c].z;
        r.red_off = at;
        r.red_cnt = red_off[c + 1] - at;
        trip[trip_off[c]] = r;
        warp = m.irr_nop[q1] > kLaneOps;
        if (!warp) triplet_images(m, q1, q2, q3, red + at);
    }
    for (unsigned left = __ballot_sync(0xffffffffu, warp); left; left &= left - 1) {
        const int l = __ffs(left) - 1;
        triplet_images_warp(m, __shfl_sync(0xffffffffu, q1, l), __shfl_sync(0xffffffffu, q2, l),
                            __shfl_sync(0xffffffffu, q3, l), red + __shfl_sync(0xffffffffu, at, l));
    }
}

__global__ void k_quartet_count(MeshDev m, const int4 *cand, int32_t n_cand, int32_t *n_q, int32_t *n_red,
                                int32_t *status) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n_cand) return;
    const int q1 = cand[c].x, q2 = cand[c].y, q3 = cand[c].z;
    int nq = 0, nr = 0;
    if (q1 < 0 || q1 >= m.n_irr || q2 < 0 || q2 >= m.n_full || q3 < 0 || q3 >= m.n_full ||
        m.irr_nop[q1] > kMaxOps) {
        atomicCAS(status, kDevOk, kDevBadIndex);
    } else if (q3 >= q2) {
        const int q4 = fourth_index(m, m.irr_full[q1], q2, q3);
        if (q4 >= q3) {
            const int k = quartet_images(m, q1, q2, q3, q4, nullptr);
            if (k >= 0) {
                nq = 1;
                nr = k;
            }
        }
    }
    n_q[c] = nq;
    n_red[c] = nr;
}

__global__ void k_quartet_fill(MeshDev m, const int4 *cand, int32_t n_cand, const int32_t *q_off,
                               const int32_t *red_off, QuartetRec *quart, int4 *red) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n_cand) return;
    if (q_off[c + 1] == q_off[c]) return;
    const int q1 = cand[c].x, q2 = cand[c].y, q3 = cand[c].z;
    const int q4 = fourth_index(m, m.irr_full[q1], q2, q3);
    const int k = quartet_images(m, q1, q2, q3, q4, red + red_off[c]);
    QuartetRec r;
    r.q1 = q1;
    r.q2 = q2;
    r.q3 = q3;
    r.q4 = q4;
    r.cand = cand[c].w;
    r.red_off = red_off[c];
    r.red_cnt = k;
    r.pad = 0;
    quart[q_off[c]] = r;
}

// ---- exclusive scan: per-block scan of 2048 elements, scan of block sums, add; up to two
// arrays at once (grid.y), and a single kernel when one block covers them ----
constexpr int kScanThreads = 1024;
constexpr int kScanItems = 2 * kScanThreads;

// in[n] to out[n + 1] (the total last); total (may be null) receives it as well.
struct Scan {
    const int32_t *in[2];
    int32_t *out[2], *total[2], *sums[2];
    int32_t n, nb;
};

// Exclusive scan over the block's threads by warp shuffles; sh holds a warp's sum each.
__device__ int32_t block_exclusive_scan(int32_t v, int32_t *sh, int32_t &total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    int32_t x = v;
    for (int o = 1; o < 32; o <<= 1) {
        const int32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sh[w] = x;
    __syncthreads();
    if (w == 0) {
        int32_t t = lane < nw ? sh[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        if (lane < nw) sh[lane] = t;
    }
    __syncthreads();
    total = sh[nw - 1];
    const int32_t before = w ? sh[w - 1] : 0;
    __syncthreads();
    return before + x - v;
}

__device__ __forceinline__ void scan_total(const Scan &a, int y, int32_t total) {
    a.out[y][a.n] = total;
    if (a.total[y]) *a.total[y] = total;
}

__global__ void k_scan_blocks(Scan a) {
    __shared__ int32_t sh[32];
    const int y = blockIdx.y;
    const int64_t i0 = (int64_t)blockIdx.x * kScanItems + 2 * threadIdx.x;
    const int32_t v = i0 < a.n ? a.in[y][i0] : 0;
    const int32_t w = i0 + 1 < a.n ? a.in[y][i0 + 1] : 0;
    int32_t total;
    const int32_t ex = block_exclusive_scan(v + w, sh, total);
    if (i0 < a.n) a.out[y][i0] = ex;
    if (i0 + 1 < a.n) a.out[y][i0 + 1] = ex + v;
    if (threadIdx.x != 0) return;
    if (a.nb == 1)
        scan_total(a, y, total);
    else
        a.sums[y][blockIdx.x] = total;
}

__global__ void k_scan_sums(Scan a) {
    __shared__ int32_t sh[32];
    const int y = blockIdx.y;
    int32_t carry = 0;
    for (int32_t c = 0; c < a.nb; c += kScanThreads) {
        const int32_t i = c + threadIdx.x;
        const int32_t v = i < a.nb ? a.sums[y][i] : 0;
        int32_t total;
        const int32_t ex = block_exclusive_scan(v, sh, total);
        if (i < a.nb) a.sums[y][i] = ex + carry;
        carry += total;
    }
    if (threadIdx.x == 0) scan_total(a, y, carry);
}

__global__ void k_scan_add(Scan a) {
    const int y = blockIdx.y;
    const int64_t i = (int64_t)blockIdx.x * kScanItems + threadIdx.x;
    const int32_t add = a.sums[y][blockIdx.x];
    if (i < a.n) a.out[y][i] += add;
    if (i + kScanThreads < a.n) a.out[y][i + kScanThreads] += add;
}

cudaError_t launch_scan(const Scan &a, int arrays, cudaStream_t s) {
    const dim3 grid((unsigned)a.nb, (unsigned)arrays);
    k_scan_blocks<<<grid, kScanThreads, 0, s>>>(a);
    if (a.nb > 1) {
        k_scan_sums<<<dim3(1, (unsigned)arrays), kScanThreads, 0, s>>>(a);
        k_scan_add<<<grid, kScanThreads, 0, s>>>(a);
    }
    return cudaGetLastError();
}

}  // namespace

namespace {
__global__ void k_build_candidates(const int4 *desc, const int32_t *list, int4 *cand) {
    const int q1 = blockIdx.y;
    const int4 d = desc[q1];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < d.y; i += gridDim.x * blockDim.x)
        cand[d.z + i] = make_int4(q1, list[d.x + i] - 1, d.w, 0);
}
}  // namespace

namespace {
// Candidates of rows that do not share one sample: per q1 the union of its rows' samples with
// the rows that hold a point as a bit mask; a point that a row holds k times gives k
// candidates, the j-th with the rows that hold it j times. cnt[r - r0][q2] counts a row's
// copies. One pass over the lists and two over (q1, q2): a few us where merging the lists on
// the host took 2.7 ms (fluorite 11^3, 216 points for each of 501 rows).
__global__ void k_union_count(int n_full, int r0, const int64_t *rbeg, const int32_t *rlen, const int32_t *list,
                              int32_t *cnt, int32_t *status) {
    const int r = r0 + blockIdx.x;
    int32_t *c = cnt + (size_t)blockIdx.x * n_full;
    for (int i = threadIdx.x; i < rlen[r]; i += blockDim.x) {
        const int32_t q2 = list[rbeg[r] + i] - 1;
        if (q2 < 0 || q2 >= n_full)
            atomicCAS(status, kDevOk, kDevBadIndex);
        else
            atomicAdd(c + q2, 1);
    }
}

// copies[q1][q2], and their sum over all q1 (64 bits) into total.
__global__ void k_union_copies(int n_full, int q0, int r0, const int32_t *row_of, const int32_t *cnt, int32_t *copies,
                               unsigned long long *total) {
    const int q1 = q0 + blockIdx.y, q2 = blockIdx.x * blockDim.x + threadIdx.x;
    int most = 0;
    if (q2 < n_full) {
        for (int r = row_of[q1]; r < row_of[q1 + 1]; ++r) most = max(most, cnt[(size_t)(r - r0) * n_full + q2]);
        copies[(size_t)q1 * n_full + q2] = most;
    }
    const int sum = __reduce_add_sync(0xffffffffu, most);
    if ((threadIdx.x & 31) == 0 && sum) atomicAdd(total, (unsigned long long)sum);
}

__global__ void k_union_write(int n_full, int q0, int r0, const int32_t *row_of, const int32_t *row_b1,
                              const int32_t *cnt, const int32_t *off, int4 *cand, uint4 *mask) {
    const int q1 = q0 + blockIdx.y, q2 = blockIdx.x * blockDim.x + threadIdx.x;
    if (q2 >= n_full) return;
    const size_t e = (size_t)q1 * n_full + q2;
    const int at = off[e], n = off[e + 1] - at;
    for (int j = 0; j < n; ++j) {
        uint32_t w[4] = {0u, 0u, 0u, 0u};
        for (int r = row_of[q1]; r < row_of[q1 + 1]; ++r)
            if (cnt[(size_t)(r - r0) * n_full + q2] > j) {
                const uint32_t b = (uint32_t)row_b1[r];
#pragma unroll
                for (int k = 0; k < 4; ++k) w[k] |= (b >> 5) == (uint32_t)k ? 1u << (b & 31) : 0u;
            }
        cand[at + j] = make_int4(q1, q2, at + j, 0);
        mask[at + j] = make_uint4(w[0], w[1], w[2], w[3]);
    }
}
}  // namespace

cudaError_t launch_union_count(int n_full, int r0, int n_row, const int64_t *rbeg, const int32_t *rlen,
                               const int32_t *list, int32_t *cnt, int32_t *status, cudaStream_t s) {
    if (n_row <= 0) return cudaSuccess;
    const cudaError_t e = cudaMemsetAsync(cnt, 0, sizeof(int32_t) * (size_t)n_row * n_full, s);
    if (e != cudaSuccess) return e;
    k_union_count<<<n_row, 256, 0, s>>>(n_full, r0, rbeg, rlen, list, cnt, status);
    return cudaGetLastError();
}

cudaError_t launch_union_copies(int n_full, int q0, int n_q1, int r0, const int32_t *row_of, const int32_t *cnt,
                                int32_t *copies, unsigned long long *total, cudaStream_t s) {
    if (n_q1 <= 0) return cudaSuccess;
    k_union_copies<<<dim3((unsigned)((n_full + 127) / 128), (unsigned)n_q1), 128, 0, s>>>(n_full, q0, r0, row_of, cnt,
                                                                                       copies, total);
    return cudaGetLastError();
}

cudaError_t launch_union_write(int n_full, int q0, int n_q1, int r0, const int32_t *row_of, const int32_t *row_b1,
                               const int32_t *cnt, const int32_t *off, int4 *cand, uint32_t *mask, cudaStream_t s) {
    if (n_q1 <= 0) return cudaSuccess;
    k_union_write<<<dim3((unsigned)((n_full + 127) / 128), (unsigned)n_q1), 128, 0, s>>>(
        n_full, q0, r0, row_of, row_b1, cnt, off, cand, reinterpret_cast<uint4 *>(mask));
    return cudaGetLastError();
}

cudaError_t launch_build_candidates(const int4 *desc, int32_t n_irr, int32_t max_len, const int32_t *list, int4 *cand,
                                    cudaStream_t s) {
    if (n_irr <= 0 || max_len <= 0) return cudaSuccess;
    dim3 grid((unsigned)((max_len + 255) / 256), (unsigned)n_irr);
    k_build_candidates<<<grid, 256, 0, s>>>(desc, list, cand);
    return cudaGetLastError();
}

size_t exclusive_scan_tmp_elems(int32_t n) { return (size_t)(n + kScanItems - 1) / kScanItems + 1; }

cudaError_t exclusive_scan_i32(const int32_t *in, int32_t *out, int32_t n, int32_t *tmp, cudaStream_t s) {
    const int32_t nb = (n + kScanItems - 1) / kScanItems;
    if (nb == 0) return cudaMemsetAsync(out, 0, sizeof(int32_t), s);
    return launch_scan(Scan{{in, nullptr}, {out, nullptr}, {nullptr, nullptr}, {tmp, nullptr}, n, nb}, 1, s);
}

cudaError_t exclusive_scan_pair_i32(const int32_t *in0, int32_t *out0, const int32_t *in1, int32_t *out1, int32_t n,
                                    int32_t *tmp, int32_t *totals, cudaStream_t s) {
    const int32_t nb = (n + kScanItems - 1) / kScanItems;
    if (nb == 0) {
        cudaError_t e = cudaMemsetAsync(out0, 0, sizeof(int32_t), s);
        if (e == cudaSuccess) e = cudaMemsetAsync(out1, 0, sizeof(int32_t), s);
        if (e == cudaSuccess) e = cudaMemsetAsync(totals, 0, 2 * sizeof(int32_t), s);
        return e;
    }
    int32_t *tmp1 = tmp + exclusive_scan_tmp_elems(n);
    return launch_scan(Scan{{in0, in1}, {out0, out1}, {totals, totals + 1}, {tmp, tmp1}, n, nb}, 2, s);
}

cudaError_t launch_triplet_count(const MeshDev &m, const int4 *cand, int32_t n_cand, int32_t *n_trip,
                                 int32_t *n_red, int32_t *status, cudaStream_t s) {
    if (n_cand <= 0) return cudaSuccess;
    k_triplet_count<<<(n_cand + 127) / 128, 128, 0, s>>>(m, cand, n_cand, n_trip, n_red, status);
    return cudaGetLastError();
}

cudaError_t launch_triplet_fill(const MeshDev &m, const int4 *cand, int32_t n_cand, const int32_t *trip_off,
                                const int32_t *red_off, TripletRec *trip, int2 *red, cudaStream_t s) {
    if (n_cand <= 0) return cudaSuccess;
    k_triplet_fill<<<(n_cand + 127) / 128, 128, 0, s>>>(m, cand, n_cand, trip_off, red_off, trip, red);
    return cudaGetLastError();
}

cudaError_t launch_quartet_count(const MeshDev &m, const int4 *cand, int32_t n_cand, int32_t *n_q,
                                 int32_t *n_red, int32_t *status, cudaStream_t s) {
    if (n_cand <= 0) return cudaSuccess;
    k_quartet_count<<<(n_cand + 127) / 128, 128, 0, s>>>(m, cand, n_cand, n_q, n_red, status);
    return cudaGetLastError();
}

cudaError_t launch_quartet_fill(const MeshDev &m, const int4 *cand, int32_t n_cand, const int32_t *q_off,
                                const int32_t *red_off, QuartetRec *quart, int4 *red, cudaStream_t s) {
    if (n_cand <= 0) return cudaSuccess;
    k_quartet_fill<<<(n_cand + 127) / 128, 128, 0, s>>>(m, cand, n_cand, q_off, red_off, quart, red);
    return cudaGetLastError();
}

}  // namespace tdg
