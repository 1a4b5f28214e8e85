// Rows of the scattering matrix and the Monte-Carlo q' samples of every row.
//
// Rows: scattering.f90:170-209 with a single rank (every (q1,b1) with omega >= lo_freqtol).
// Random stream: lo_randomnumbers.f90:203-273. TDEP seeds MT19937-64 with
// init_genrand64 and draws genrand64_real1: the generator of Nishimura and Matsumoto (2000),
// here a block of 312 words at a time so that the recurrence and the tempering vectorise.
// Samples: lo_fftgrid_helper.f90:56-99 (mc_point_to_full, generate_grid).
#pragma GCC optimize("O3")  // the generator's loops vectorise
#include <algorithm>
#include <cstring>
#include <vector>

#include "../../../include/tdep_gb300.h"
#include "crystal.hpp"

namespace tdg {
namespace {

struct McGrid {
    int mc[3], full[3];
    double ratio[3];
    int npoints;
};

McGrid make_grid(const int32_t full[3], const int32_t mc[3]) {
    McGrid g;
    for (int i = 0; i < 3; ++i) {
        g.full[i] = full[i];
        g.mc[i] = std::min(mc[i], full[i]);
        g.ratio[i] = (double)g.full[i] / (double)g.mc[i];
    }
    g.npoints = g.mc[0] * g.mc[1] * g.mc[2];
    return g;
}

class Mt64 {
  public:
    static constexpr int kN = 312;
    explicit Mt64(uint64_t word) {
        s_[0] = word;
        for (int i = 1; i < kN; ++i) s_[i] = 6364136223846793005ULL * (s_[i - 1] ^ (s_[i - 1] >> 62)) + (uint64_t)i;
        at_ = kN;
    }
    // The generator with block `state` in hand, its words before `at` taken.
    Mt64(const uint64_t *state, int at) : at_(at) {
        std::memcpy(s_, state, sizeof s_);
        temper(s_, t_, kN);
    }
    uint64_t next() {
        if (at_ == kN) {
            refill();
            temper(s_, t_, kN);
            at_ = 0;
        }
        return t_[at_++];
    }
    const uint64_t *state() const { return s_; }
    int taken() const { return at_; }
    // The next block of the recurrence.
    void refill() {
        for (int i = 0; i < kM; ++i) s_[i] = twist(s_[i], s_[i + 1], s_[i + kM]);
        for (int i = kM; i < kN - 1; ++i) s_[i] = twist(s_[i], s_[i + 1], s_[i - kM]);
        s_[kN - 1] = twist(s_[kN - 1], s_[0], s_[kM - 1]);
    }
    static uint64_t temper(uint64_t x) {
        x ^= (x >> 29) & 0x5555555555555555ULL;
        x ^= (x << 17) & 0x71D67FFFEDA60000ULL;
        x ^= (x << 37) & 0xFFF7EEE000000000ULL;
        return x ^ (x >> 43);
    }

  private:
    static constexpr int kM = 156;
    static uint64_t twist(uint64_t hi, uint64_t lo, uint64_t far) {
        const uint64_t x = (hi & 0xFFFFFFFF80000000ULL) | (lo & 0x7FFFFFFFULL);
        return far ^ (x >> 1) ^ ((0 - (x & 1ULL)) & 0xB5026F5AA96619E9ULL);
    }
    static void temper(const uint64_t *s, uint64_t *t, int n) {
        for (int i = 0; i < n; ++i) t[i] = temper(s[i]);
    }
    uint64_t s_[kN], t_[kN];
    int at_;
};

// genrand64_real1: 53-bit integer on [0,1] inclusive.
double real1(Mt64 &rng) { return (double)(rng.next() >> 11) * (1.0 / (9007199254740992.0 - 1.0)); }

// One point of the cell gm (1-based) of the Monte-Carlo grid.
int mc_point_to_full(const McGrid &g, const int gm[3], Mt64 &rng) {
    int gf[3];
    for (int d = 0; d < 3; ++d) gf[d] = (int)std::ceil(((double)gm[d] - 1.0) * g.ratio[d] + real1(rng) * g.ratio[d]);
    return (gf[0] - 1) * g.full[1] * g.full[2] + (gf[1] - 1) * g.full[2] + gf[2];
}

// A row's sample, cell after cell (last index fastest), never the point just drawn again.
void draw_grid(const McGrid &g, int32_t *out, Mt64 &rng) {
    int32_t *o = out;
    int qprev = 0;
    for (int i = 1; i <= g.mc[0]; ++i)
        for (int j = 1; j <= g.mc[1]; ++j)
            for (int k = 1; k <= g.mc[2]; ++k) {
                const int gm[3] = {i, j, k};
                int q = mc_point_to_full(g, gm, rng);
                while (o != out && q == qprev) q = mc_point_to_full(g, gm, rng);
                *o++ = q;
                qprev = q;
            }
}

// Samples of rows [0, n_row) on a Monte-Carlo grid that is the mesh. A cell is then one point,
// which every draw r in (0, 1] gives, ceil((gm - 1) + r) = gm, except where r is so small
// that the sum rounds to gm - 1: below 2^-40 for up to 4096 points a side. So the samples are
// the mesh in order unless some draw is below that; the words are drawn all the same, blocks
// of them by the recurrence in this thread (the part that is a chain), tempered and looked
// at on all threads. Returns the rows that are done and leaves rng at the next one's start:
// all rows, but for one draw in 10^12. (Drawn point by point, the two million points of a
// five-atom 12^3 mesh took 30 ms.)
// low: 2^24 as a word, 2^-40 as a draw.
int mesh_samples(const McGrid &g, int n_row, int32_t *list, Mt64 &rng, uint64_t low_word) {
    const int64_t words = 3 * (int64_t)g.npoints;
    const int batch = (int)std::max<int64_t>(1, (1 << 18) / words);
    constexpr int kN = Mt64::kN;
    std::vector<uint64_t> blocks;
    for (int r0 = 0; r0 < n_row; r0 += batch) {
        const int nr = std::min(batch, n_row - r0);
        const int at = rng.taken();
        const int64_t nb = (at + nr * words + kN - 1) / kN;  // the block in hand first
        blocks.resize((size_t)(nb * kN));
        std::memcpy(blocks.data(), rng.state(), sizeof(uint64_t) * kN);
        for (int64_t b = 1; b < nb; ++b) {
            rng.refill();
            std::memcpy(blocks.data() + b * kN, rng.state(), sizeof(uint64_t) * kN);
        }
        std::vector<char> low(nr, 0);
        parallel_for(nr, [&](int64_t r) {
            const uint64_t *w = blocks.data() + at + r * words;
            uint64_t hit = 0;
            for (int64_t i = 0; i < words; ++i) hit |= (uint64_t)(Mt64::temper(w[i]) < low_word);
            low[r] = hit != 0;
            int32_t *out = list + (r0 + r) * (int64_t)g.npoints;
            for (int q = 0; q < g.npoints; ++q) out[q] = q + 1;
        });
        int done = 0;
        while (done < nr && !low[done]) ++done;
        const int64_t next = at + done * words;
        // the block that holds the next word, or the last one with all its words taken
        const int64_t b = std::min(next / kN, nb - 1);
        rng = Mt64(blocks.data() + b * kN, (int)(next - b * kN));
        if (done < nr) return r0 + done;
    }
    return n_row;
}

// The samples of n_row rows on a grid that is the mesh, rows with a low draw point by point.
constexpr uint64_t kLowWord = (uint64_t)1 << 24;
void mesh_lists(const McGrid &g, int n_row, int32_t *list, Mt64 &rng, uint64_t low_word) {
    for (int first = 0; first < n_row;) {
        first += mesh_samples(g, n_row - first, list + (size_t)first * g.npoints, rng, low_word);
        if (first < n_row) {
            draw_grid(g, list + (size_t)first * g.npoints, rng);
            ++first;
        }
    }
}

}  // namespace

// 64-bit seed word of init_genrand64(iseed=0, rseed=1/seed).
uint64_t tdep_seed_word(int seed) {
    const double rseed = 1.0 / (double)seed;
    const double f0 = rseed - std::floor(rseed) - 0.5;
    const int64_t s = (int64_t)anint(f0 * 1073741824.0);
    return (uint64_t)s;
}

}  // namespace tdg

extern "C" int tdg_mc_qlists(const tdg_problem *p, const tdg_opts *o, int32_t *n_row, int32_t *row_q1,
                             int32_t *row_b1, int64_t *ptr3, int32_t *list3, int64_t *ptr4, int32_t *list4a,
                             int32_t *list4b) {
    using namespace tdg;
    if (!p || !o || !n_row || !row_q1 || !row_b1) return set_error(kErrParam, "tdg_mc_qlists: null argument");
    if (o->seed <= 0) return set_error(kErrParam, "tdg_mc_qlists: seed must be positive");
    const int nb = p->n_mode;
    int nr = 0;
    for (int q1 = 0; q1 < p->n_irr; ++q1) {
        const int f = p->irr_full[q1] - 1;
        for (int b1 = 0; b1 < nb; ++b1) {
            if (p->omega[(size_t)f * nb + b1] < kFreqTol) continue;
            row_q1[nr] = q1 + 1;
            row_b1[nr] = b1 + 1;
            ++nr;
        }
    }
    *n_row = nr;
    Mt64 rng(tdep_seed_word(o->seed));
    const McGrid g3 = make_grid(p->grid, o->qg3ph);
    const McGrid g4 = make_grid(p->grid, o->qg4ph);
    if (o->thirdorder && (!ptr3 || !list3)) return set_error(kErrParam, "tdg_mc_qlists: missing third-order lists");
    if (o->fourthorder && (!ptr4 || !list4a || !list4b))
        return set_error(kErrParam, "tdg_mc_qlists: missing fourth-order lists");
    if (ptr3) ptr3[0] = 0;
    if (ptr4) ptr4[0] = 0;
    // rows take their three- and four-phonon samples in turn from one stream
    int first = 0;
    bool mesh3 = o->thirdorder && !o->fourthorder;
    for (int d = 0; d < 3; ++d) mesh3 = mesh3 && g3.mc[d] == g3.full[d] && g3.full[d] <= 4096;
    for (int r = 0; r < nr; ++r) {
        if (o->thirdorder) ptr3[r + 1] = (int64_t)(r + 1) * g3.npoints;
        if (o->fourthorder) ptr4[r + 1] = (int64_t)(r + 1) * g4.npoints;
    }
    if (mesh3) {
        mesh_lists(g3, nr, list3, rng, kLowWord);
        first = nr;
    }
    for (int r = first; r < nr; ++r) {
        if (o->thirdorder) draw_grid(g3, list3 + (size_t)r * g3.npoints, rng);
        if (o->fourthorder) {
            draw_grid(g4, list4a + (size_t)r * g4.npoints, rng);
            draw_grid(g4, list4b + (size_t)r * g4.npoints, rng);
        }
    }
    return kOk;
}

extern "C" int tdg_check_mesh_samples(const int32_t grid[3], int32_t seed, int32_t n_row, uint64_t low_word,
                                      int32_t *list, uint64_t next[8]) {
    using namespace tdg;
    if (!grid || !list || !next || n_row < 0 || grid[0] < 1 || grid[1] < 1 || grid[2] < 1 || grid[0] > 4096 ||
        grid[1] > 4096 || grid[2] > 4096 || seed <= 0)
        return set_error(kErrParam, "tdg_check_mesh_samples: bad argument");
    Mt64 rng(tdep_seed_word(seed));
    mesh_lists(make_grid(grid, grid), n_row, list, rng, low_word);
    for (int i = 0; i < 8; ++i) next[i] = rng.next();
    return kOk;
}
