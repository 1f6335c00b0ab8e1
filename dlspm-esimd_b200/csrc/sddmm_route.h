// Which SDDMMs run on the tensor cores (sddmm_mma.cuh) and which on the gather kernels: estimates of both times from the
// sizes of a call.  Host code without CUDA.
//
// All times are in microseconds, measured on a B200 with operands in L2 or, for large groups, in memory.
#pragma once
#include <math.h>

#include <algorithm>
#include <vector>

namespace dlspm {

constexpr int kPickInner = 64;  // of the inner dimension per stage, and per main accumulator
constexpr int kPickCols = 128;  // columns of the pattern per block, 256 per pair
constexpr int kPickRows = 64;   // rows of the pattern converted per block at most, 128 per pair
constexpr int kPickCheckMost = 8192;  // problems of a launch at most

struct SddmmSizes {
    int M, K, N;  // N: inner dimension
    double nnz;
    bool masked;  // factors of the entries
    bool wide;    // rows of lhs and rhs allow 16-byte loads
    double density() const { return nnz / ((double)M * K); }
};

inline long long route_ceil(long long a, long long b) { return (a + b - 1) / b; }

// ---- tensor cores -------------------------------------------------------------------------------------------------

// Byte offsets into the operands are 32-bit in the kernel (and run up to a strip past the end).  Problems of up to three
// strips stay with the gather kernels.
inline bool pick_takes(const SddmmSizes &q)
{
    return q.nnz > 0 && q.M > 3 * 2 * kPickRows && q.K > 0 && q.N > 0 && ((double)std::max(q.M, q.K) + 512) * q.N < 1e9;
}

// Factors of the entries are read between a look-up and its store: this much per row and unit of density of a tile.  0.10
// to 0.25 while the entries' arrays stay in L2 (4096 x 4096 at 30 %: 20 MB each), 0.25 to 0.4 from 8 million entries on;
// in a grouped call the other problems' arrays are there as well.
inline double pick_factor_us(const SddmmSizes &q, bool grouped) { return !q.masked ? 0.0 : grouped || q.nnz > 6e6 ? 0.35 : 0.2; }

// A tile of `rows` rows: the look-ups with some of the conversions (64 of the inner dimension each) beside them, or the
// conversions alone.  A conversion waits longer for its numbers in a grouped call, where every pair of blocks reads an
// rhs of its own (37 problems of 1024 x 4096, inner dimension 256, at 10 % nonzeros: 10.7 us a tile; one pattern of 8192 x
// 4096: 7.3), and with loads of less than 16 bytes.  Fitted to 389 to 16384 rows, 2 to 50 % nonzeros, inner dimensions 16
// to 800; root mean square of the relative error over 450 lone calls 5 %, over 440 grouped ones 8 %.
inline double pick_tile_us(const SddmmSizes &q, int rows, bool grouped)
{
    const double steps = (double)route_ceil(q.N, kPickInner) * (q.wide ? 1.0 : 1.14);
    const double look_ups = (5.9 + 25.0 * q.density()) * (0.25 + 0.75 * rows / (2 * kPickRows)) + pick_factor_us(q, grouped) * rows * q.density();
    return std::max(look_ups + (grouped ? 0.74 : 0.62) * steps, (grouped ? 1.87 : 1.48) * steps);
}

// A pattern on its own: rows per strip and parts of a strip so that the rounds of strips over the pairs of blocks end
// together.
struct PickShape {
    int strip_rows, parts;
    double us;
};
inline PickShape pick_shape(int sm_count, const SddmmSizes &q)
{
    const int pairs = sm_count / 2, tiles = (int)route_ceil(q.K, 2 * kPickCols);
    PickShape best = {2 * kPickRows, 1, 1e30};
    for (int rows = 2 * kPickRows; rows >= 32; rows -= 16) {
        const double tile_us = pick_tile_us(q, rows, false);
        for (int s = 1; s <= 2 && s <= tiles; s++) {
            const double us = 5.5 + (double)route_ceil(route_ceil(q.M, rows) * s, pairs) * ((double)route_ceil(tiles, s) * tile_us + 3.2 + 4.0 * (s - 1));
            if (us < best.us - 1e-9) best = {rows, s, us};
        }
    }
    return best;
}

// A pattern on its own, against the gather kernels at rates that few patterns exceed (even rows, dense; uneven rows are
// slower) and with a margin for the errors of the estimates.  Measured, gather / tensor cores, taken: 8192 x 4096, inner
// dimension 256, at 10 % 180 / 158; 2048 x 512, 256, at 50 % 30 / 27; 1024 x 4096, 512, at 30 % 161 / 100; left alone: 8192
// x 4096, 256, at 2 % 39 / 127; 8192 x 8192, 64, at 10 % 92 / 188; 1024 x 4096, 128, at 50 % 65 / 80; 573 x 3711, 71, at
// 50 % 43 / 77.  Of 1200 calls of 64 to 16384 rows none that was taken was slower for it.
inline bool pick_pays_alone(int sm_count, const SddmmSizes &q)
{
    if (!pick_takes(q)) return false;
    const double rate = !q.wide ? 4.0 : q.N <= 64 ? 9.0 : q.N <= 128 ? 9.5 : 9.3 + 3.0 * q.density();
    return pick_shape(sm_count, q).us < (q.masked ? 0.9 : 0.95) * (4.0 + 2.0 * q.nnz * q.N / (rate * 1e6));
}

// A problem of a grouped call: rows per strip, strips, and the parts of each.  Long strips are cut into up to four parts,
// so that no pair of blocks is left with one at the end.
struct PickCut {
    int strip_rows, strips, parts;
};
inline PickCut pick_cut(const SddmmSizes &q)
{
    const long long most = route_ceil(q.M, 2 * kPickRows), tiles = route_ceil(q.K, 2 * kPickCols);
    PickCut c;
    c.strip_rows = (int)route_ceil(route_ceil(q.M, most), 16) * 16;
    c.strips = (int)route_ceil(q.M, c.strip_rows);
    c.parts = (int)std::max(1LL, std::min({4LL, tiles, (long long)((double)tiles * pick_tile_us(q, 2 * kPickRows, true) / 80.0) + 1}));
    return c;
}

// Part `part` of a strip: the pair's tiles, and the search for where the part begins and ends in every row.
inline double pick_part_us(const SddmmSizes &q, const PickCut &c, int part)
{
    const long long tiles = route_ceil(q.K, kPickCols);
    const auto boundary = [&](int b) { return tiles * b / (2 * c.parts); };
    const int b = 2 * part;
    const long long most = std::max(boundary(b + 1) - boundary(b), boundary(b + 2) - boundary(b + 1));
    return 2.7 + (c.parts > 1 ? 2.5 * (b + 1) : 0.0) + (double)most * pick_tile_us(q, c.strip_rows, true);
}

// Order of the problems in a grouped launch: the longest strips first, which are dealt to the pairs of blocks in turn.
inline double pick_order(const SddmmSizes &q, const PickCut &c) { return (double)q.K / c.parts * (q.N + kPickInner); }

// A launch over problems of a grouped call: the longest pair of the deal.
inline double pick_group_us(int sm_count, const std::vector<SddmmSizes> &problems)
{
    struct Entry {
        SddmmSizes q;
        PickCut c;
    };
    std::vector<Entry> tab;
    for (const SddmmSizes &q : problems) tab.push_back(Entry{q, pick_cut(q)});
    std::stable_sort(tab.begin(), tab.end(), [](const Entry &x, const Entry &y) { return pick_order(x.q, x.c) > pick_order(y.q, y.c); });
    const int pairs = sm_count / 2;
    std::vector<double> busy((size_t)pairs, 0.0);
    int at = 0;
    for (const Entry &e : tab) {
        double us[4], strip = 0.0;
        for (int part = 0; part < e.c.parts; part++) strip += us[part] = pick_part_us(e.q, e.c, part);
        // (whole rounds of very many strips at once)
        const int rounds = std::max(0, e.c.strips / pairs - 16), rest = e.c.strips - rounds * pairs;
        for (double &b : busy) b += rounds * strip;
        for (int i = 0; i < rest; i++)
            for (int part = 0; part < e.c.parts; part++) {
                busy[(size_t)at] += us[part];
                at = at + 1 == pairs ? 0 : at + 1;
            }
    }
    return *std::max_element(busy.begin(), busy.end());
}

// ---- gather kernels of a grouped call --------------------------------------------------------------------------------

// Class of a problem whose rows allow 128-bit loads, one launch each: the register-resident layouts of sddmm_layout (1 to
// 5), segments of 1024 floats beyond them and of 512 from N = 2052 on (the choice of the single-matrix launcher), and rows
// of up to 16 and 32 floats in groups of four lanes, as there.
inline int sddmm_class(int N)
{
    return N <= 16 ? 10 : N <= 32 ? 11 : N <= 64 ? 1 : N <= 128 ? 2 : N <= 256 ? 3 : N <= 512 ? 4 : N <= 1024 ? 5 : N <= 2048 ? 6 : 7;
}

// Most warps per row (as a shift) in a class of `rows` rows.
inline int sharing_most(int sm_count, long long rows)
{
    const long long want = (long long)sm_count * 32;
    if (rows * 4 >= want * 3) return 0;
    int shift = 0;
    while (shift < 3 && (rows << shift) < want) shift++;
    return shift;
}
// The same for one problem of it whose rows have `mean` entries (register-resident rows).
inline int sharing_shift(int most, double mean)
{
    int s = 0;
    while (s < most && mean > 32.0 * (1 << s)) s++;
    return s;
}

// TFLOP/s where a call fills the device (the higher of what was measured), and microseconds per entry of a row that a single warp walks, which is what
// bounds a class with few rows (1024 rows of 2000 entries in a class of 4736 rows, inner dimension 256: 709 us).
inline double gather_rate(int N) { return N <= 32 ? 6.5 : N <= 64 ? 7.6 : N <= 128 ? 10.5 : 12.0; }
inline double gather_entry_us(int N) { return N <= 64 ? 0.045 : N <= 128 ? 0.054 : N <= 256 ? 0.0006 * N : 0.0768 + 0.0003 * N; }

// The gather kernels over problems of a call: the classes run side by side, so together they take as long as their work,
// and each as long as its longest row.  That row is taken as the mean one of its problem: right for even rows, too low a
// figure for uneven ones, whose spread is not known here (rows with a spread of 40 %: 30 % too short a time on average).
inline double gather_group_us(int sm_count, const std::vector<SddmmSizes> &problems)
{
    long long rows[12] = {};
    double work = 0.0, longest = 0.0;
    for (const SddmmSizes &q : problems) {
        rows[sddmm_class(q.N)] += q.M;
        work += 2.0 * q.nnz * q.N / (gather_rate(q.N) * 1e6);
    }
    if (work == 0.0) return 0.0;
    for (const SddmmSizes &q : problems) {
        const double mean = q.nnz / q.M;
        longest = std::max(longest, mean / (1 << sharing_shift(sharing_most(sm_count, rows[sddmm_class(q.N)]), mean)) * gather_entry_us(q.N));
    }
    return 20.0 + pow(pow(work, 1.83) + pow(longest, 1.83), 1.0 / 1.83);
}

// Which problems of a grouped call go to the tensor cores: those for which they are the cheaper way on a full device, if
// the call as a whole (that launch, then the gather of the others) is then faster than gathering everything.  The factors
// cover the errors of the estimates.  Measured on 360 calls of 8 to 150 problems, half of them with even rows and half
// with a spread of 40 %: 183 are split, and take 0.3 to 1.02 of the time of the gather alone.  (With the estimates at face
// value 226 are split, and some take up to 1.2 of it.)
inline void sddmm_route_group(int sm_count, const std::vector<SddmmSizes> &problems, unsigned char *chosen)
{
    std::vector<SddmmSizes> dense, rest, all;
    for (size_t i = 0; i < problems.size(); i++) {
        const SddmmSizes &q = problems[i];
        chosen[i] = 0;
        if (q.M <= 0 || q.N <= 0 || q.nnz <= 0 || !q.wide) continue;  // (run one by one, whatever is chosen)
        if (pick_takes(q)) {
            const PickCut c = pick_cut(q);
            double strip = 0.0;
            for (int part = 0; part < c.parts; part++) strip += pick_part_us(q, c, part);
            chosen[i] = c.strips * strip / (sm_count / 2) < 2.0 * q.nnz * q.N / 9.8e6;
        }
        all.push_back(q);
        (chosen[i] ? dense : rest).push_back(q);
    }
    if (dense.empty()) return;
    if ((int)dense.size() > kPickCheckMost ||
        1.1 * pick_group_us(sm_count, dense) + gather_group_us(sm_count, rest) >= 0.95 * gather_group_us(sm_count, all))
        std::fill(chosen, chosen + problems.size(), (unsigned char)0);
}

}  // namespace dlspm
