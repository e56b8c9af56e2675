// overlap.cuh -- one random-overlap pass of two k-distributions on one warp
// (radtran/cirsradg/noverlapg.f:110-147, 175-190 with rankg.f:59-152).
//
// Lane g holds ordinate g of both distributions.  An element of the combined
// distribution travels as one 32-bit word; the words are sorted in registers
// (up to 256 elements) or by merging the NG rows of keys A(i) + B(j), which are
// in order when B is monotone, in shared memory.  The cumulative weights come
// from a warp scan, and lane b then walks bin b in the sorted order.
//
// What bounds it: instruction issue (2.6 of 4 per cycle and SM with 24 warps) and
// the latency of shared memory and shuffles.  120 layers, 4 absorbers, 2000
// wavenumbers (720000 passes of 400 keys, a third of them with rows already in
// order): the forward kernel takes 3.27 ms, 3265 warp instructions a pass.  With
// the merge on 64-bit words of key and element, and weights and columns in
// shared-memory tables, it took 5.45 ms (4575 instructions and 585 bank
// conflicts a pass); with the 400 words sorted in 16 registers a lane it takes 3.69 ms.
#pragma once
#include <stdint.h>

#include <algorithm>

#include "quotient.h"
#include "rtb_common.h"

namespace rtb {

constexpr unsigned kFull = 0xffffffffu;

// An element (i, j) of a pass in one 32-bit word: i << 5 | j in the low ten
// bits, above them the leading bits of key - smallest key.  kEnd lies above
// every word of the merge; the register sort compares words as positive floats,
// with kPad above them all.  The element kIdMask names lane 31, whose weight is
// zero.
constexpr unsigned kIdBits = 10;
constexpr unsigned kIdMask = (1u << kIdBits) - 1;
constexpr unsigned kEnd = 0xffffffffu;
constexpr unsigned kPad = 0x7f7fffffu;      // the largest finite float

__device__ __forceinline__ float wkey(unsigned long long w) { return __uint_as_float((unsigned)(w >> 32)); }

// NR heapsort of radtran/cirsradg/sort2g.f:1-52 on 64-bit words (float bits of
// RA << 32 | IB) in shared memory, one thread: the comparisons are the float
// comparisons of sort2g.f (RA(J) < RA(J+1), RRA < RA(J)), so the words end in
// exactly its order.  The sift-down loads the four grandchildren while it
// compares the two children, so that no shared-memory load is on the critical
// path of a level.
static __device__ __noinline__ void heapsort_words(int n, unsigned long long* W0) {
    if (n < 2) return;
    unsigned long long* W = W0 - 1;            // W[1..n]
    int L = n / 2 + 1, IR = n;
    for (;;) {
        unsigned long long R;
        if (L > 1) {
            L = L - 1;
            R = W[L];
        } else {
            R = W[IR];
            W[IR] = W[1];
            IR = IR - 1;
            if (IR == 1) {
                W[1] = R;
                return;
            }
        }
        const float kR = wkey(R);
        int I = L, J = L + L;
        if (J <= IR) {
            unsigned long long c0 = W[J], c1 = W[J < IR ? J + 1 : J];
            for (;;) {
                // grandchildren of J and J + 1 (clamped into 1..IR; used only when in range)
                const int G = J + J;
                const unsigned long long g0 = W[G <= IR ? G : IR], g1 = W[G + 1 <= IR ? G + 1 : IR];
                const unsigned long long g2 = W[G + 2 <= IR ? G + 2 : IR], g3 = W[G + 3 <= IR ? G + 3 : IR];
                int Jc = J;
                unsigned long long c = c0;
                if (J < IR && wkey(c0) < wkey(c1)) {
                    Jc = J + 1;
                    c = c1;
                }
                if (!(kR < wkey(c))) break;
                W[I] = c;
                I = Jc;
                J = Jc + Jc;
                if (J > IR) break;
                c0 = Jc == G / 2 ? g0 : g2;
                c1 = Jc == G / 2 ? g1 : g3;
            }
        }
        W[I] = R;
    }
}

constexpr int kMergeLevels = 5;   // merge levels of NG <= 32 rows

// What a lane does at one merge level, for NG rows (run = NG << level).  Pair p
// of runs (start st_p of n = NG^2) is served by lanes [L_p, L_p+1), L_p =
// floor(32 st_p / n), which split it evenly: no lane's output range crosses a
// pair, so every lane runs a single merge per level (14 steps for NG = 20).
// Byte offsets: a and b the pair's runs in the source (b the kEnd after a where
// there is no right run), diag of the range's first position in the pair, out
// the range in the target; [lo, hi] what the bisection for the left run's share
// starts from; len words.
struct MergeLane {
    unsigned short a, b, diag, lo, hi, out, len, pad;
};
inline MergeLane merge_lane(int ng, int level, int l) {   // on the host, once per set of tables
    const int n = ng * ng, run = ng << level;
    MergeLane M = {0, 0, 0, 0, 0, 0, 0, 0};
    if (run >= n) return M;
    const int two = run << 1, npairs = (n + two - 1) / two;
    using std::max;
    using std::min;
    auto start = [&](int q) {                  // first output position of lane q
        if (q >= 32) return n;
        int p = 0;
        while (p + 1 < npairs && (32 * (p + 1) * two) / n <= q) ++p;
        const int st = p * two, sz = min(two, n - st);
        const int lp = (32 * st) / n, lq = p + 1 < npairs ? (32 * (p + 1) * two) / n : 32;
        return st + ((q - lp) * sz) / (lq - lp);
    };
    const int s = start(l), e = start(l + 1), p = s / two, ms = p * two;
    if (s >= e) return M;
    const int m = min(run, n - ms), ny = max(0, min(run, n - ms - run)), kk = s - ms;
    M.a = (unsigned short)(4 * (2 * p * (run + 1)));
    M.b = (unsigned short)(M.a + 4 * (ny > 0 ? run + 1 : m));
    M.diag = (unsigned short)(4 * kk);
    M.lo = (unsigned short)(4 * max(0, kk - ny));
    M.hi = (unsigned short)(4 * min(kk, m));
    M.out = (unsigned short)(two >= n ? 8 * s + 4 : 4 * (p * (two + 1) + kk));
    M.len = (unsigned short)(e - s);
    return M;
}

__device__ __forceinline__ unsigned lds32(unsigned at) {
    unsigned v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(at) : "memory");
    return v;
}

// One step of a merge on shared-memory byte addresses: the smaller of the two
// front words to `out`, the next word of its run in its place.  Words differ,
// and the kEnd after a run is never written out while the other run has words.
__device__ __forceinline__ void merge_step(unsigned& x, unsigned& y, unsigned& pa, unsigned& pb, unsigned out) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .u32 o;\n\t"
        "setp.lt.u32 p, %0, %1;\n\t"
        "min.u32 o, %0, %1;\n\t"
        "@p add.u32 %2, %2, 4;\n\t"
        "@!p add.u32 %3, %3, 4;\n\t"
        "st.shared.u32 [%4], o;\n\t"
        "@p ld.shared.u32 %0, [%2];\n\t"
        "@!p ld.shared.u32 %1, [%3];\n\t}"
        : "+r"(x), "+r"(y), "+r"(pa), "+r"(pb)
        : "r"(out)
        : "memory");
}

// Sorts ng sorted rows of ng words, row i at i (ng + 1) with kEnd after it in
// the buffer `from`, through `gd` and `rec` in turn; the last level reads gd and
// writes the words of the records (rec[p].y, position p).  A level merges pairs
// of runs of length run into runs of 2 run, each followed by kEnd: every lane
// finds by bisection where its output range (mtab) starts in the pair's two
// runs and merges from there.  Shared-memory byte addresses.
template <int NGC>
__device__ __forceinline__ void merge_rows(unsigned gd, unsigned rec, const MergeLane* mtab, int ng_run, int levels, int lane) {
    const int ng = NGC ? NGC : ng_run, n = ng * ng;
    unsigned from = (levels & 1) ? gd : rec;
#pragma unroll 1
    for (int level = 0; level < levels; ++level) {
        const uint4 d = *(const uint4*)(mtab + level * 32 + lane);
        const unsigned A = from + (d.x & 0xffffu), Bv = from + (d.x >> 16) + (d.y & 0xffffu);
        unsigned lo = d.y >> 16, hi = d.z & 0xffffu;
        while (lo < hi) {
            const unsigned mid = ((lo + hi) >> 1) & ~3u;
            if (lds32(A + mid) < lds32(Bv - 4 - mid)) lo = mid + 4; else hi = mid;
        }
        unsigned pa = A + lo, pb = Bv - lo;
        unsigned x = lds32(pa), y = lds32(pb);
        const bool last = level + 1 == levels;
        const unsigned to = gd + rec - from, step = last ? 8u : 4u;
        unsigned out = to + (d.z >> 16);
        const unsigned end = out + step * (d.w & 0xffffu);
#pragma unroll 2
        for (; out < end; out += step) merge_step(x, y, pa, pb, out);
        const int two = ng << (level + 1);
        if (!last && lane * two < n) {
            const unsigned at = to + 4 * (lane * (two + 1) + min(two, n - lane * two));
            asm volatile("st.shared.u32 [%0], %1;" ::"r"(at), "r"(kEnd) : "memory");
        }
        __syncwarp();
        from = to;
    }
}

__device__ __forceinline__ void order(float& a, float& b) {
    const float lo = fminf(a, b);
    b = fmaxf(a, b);
    a = lo;
}

// Sorts the 32 * E words of a warp (positive finite floats) ascending over
// (lane, register).  Each lane's words are sorted first by Batcher's network,
// then by bitonic merges over 2, 4, .. 32 lanes.  A lane that keeps the larger
// word of an exchange holds its words negated during it, so that every
// exchange is one minimum with the negated partner: the sign changes run on
// the FMA pipe, the minima on the half-rate ALU pipe, which bounds the sort.
template <int E>
__device__ __forceinline__ void warp_sort(float (&x)[E], int lane) {
#pragma unroll
    for (int p = 1; p < E; p <<= 1)
#pragma unroll
        for (int k = p; k >= 1; k >>= 1)
#pragma unroll
            for (int j = k % p; j + k < E; j += 2 * k)
#pragma unroll
                for (int i = 0; i < k; ++i)
                    if (j + i + k < E && (j + i) / (2 * p) == (j + i + k) / (2 * p)) order(x[j + i], x[j + i + k]);
#pragma unroll 1
    for (int m = 1; m < 32; m <<= 1) {
        float s = (lane & m) ? -1.0f : 1.0f;
        float y[E];
#pragma unroll
        for (int e = 0; e < E; ++e) x[e] *= s;
#pragma unroll
        for (int e = 0; e < E; ++e) y[e] = __shfl_xor_sync(kFull, x[E - 1 - e], 2 * m - 1);
#pragma unroll
        for (int e = 0; e < E; ++e) x[e] = fminf(x[e], -y[e]);
#pragma unroll 1
        for (int d = m >> 1; d >= 1; d >>= 1) {
            const float s2 = (lane & d) ? -1.0f : 1.0f, f = s * s2;
            s = s2;
#pragma unroll
            for (int e = 0; e < E; ++e) x[e] *= f;
#pragma unroll
            for (int e = 0; e < E; ++e) x[e] = fminf(x[e], -__shfl_xor_sync(kFull, x[e], d));
        }
#pragma unroll
        for (int e = 0; e < E; ++e) x[e] *= s;
#pragma unroll
        for (int k = E / 2; k >= 1; k >>= 1)
#pragma unroll
            for (int e = 0; e < E; ++e)
                if (!(e & k)) order(x[e], x[e | k]);
    }
}

// Scratch of one warp's pass, in sorted order: the elements' records and the
// FP64 prefix of the weights over each lane's chunk (the positions from NG * NG
// on are pads).  Both also take the merge's runs, and gd the heapsort's words and
// the sequential walk's new columns.
struct PassScratch {
    double* gd;        // [32 * chunk]
    uint2* rec;        // [32 * chunk + 1]: {key * weight, word}; the last one an empty element
    const MergeLane* mtab;   // [level][lane], of the CTA
    float* col;        // [column][NG]: the mix's gas columns
    float2* kg;        // [gas with a table][NG]: k and dk/dT of the layer's gases
};
__host__ __device__ constexpr int pass_chunk(int ng) { return (ng * ng + 31) / 32; }
// gd and rec each hold NG rows of NG + 1 words, and gd the sequential walk's kMaxCols
// rows of 32: up to NG 9 those are the most.  Rows of NG words, and rankk's arrays at
// offsets by NG, would need no more than the elements, but the passes' instances lose
// by it: 10-point tables, 73 layers, 3 absorbers, 515 wavenumbers took 292 us with
// them, 276 so.
__host__ __device__ constexpr int pass_gd_bytes(int ng) {
    const int pref = 8 * 32 * pass_chunk(ng), rows = (4 * ng * (ng + 1) + 15) & ~15, cols = 4 * 32 * kMaxCols;
    return pref > rows ? (pref > cols ? pref : cols) : (rows > cols ? rows : cols);
}
__host__ __device__ constexpr int pass_kg_offset(int ng) { return 2 * pass_gd_bytes(ng) + 16; }
__host__ __device__ constexpr int pass_scratch_bytes(int ng, int ncol, int ngk) {
    return (pass_kg_offset(ng) + 8 * ngk * ng + 4 * ncol * ng + 15) & ~15;
}

// The same scratch as the work arrays of rankk, at offsets in 32-bit words: value,
// derivative and weight of its 2 NG elements, 2 NG + 1 words of work, k and dk/dT of
// the NG bins, the elements' order in 16 bits.
struct RankkOff {
    static constexpr int cont = 0, dcont = 2 * kMaxNg, fac = 4 * kMaxNg, tmp = 6 * kMaxNg, kg = 8 * kMaxNg + 2,
                         dkg = kg + kMaxNg, ico = dkg + kMaxNg;
    static constexpr int bytes(int ng) { return 4 * ico + 2 * 2 * ng; }
};
constexpr bool scratch_fits() {
    for (int ng = kNgMin; ng <= kNgMax; ++ng)
        if (RankkOff::bytes(ng) > pass_scratch_bytes(ng, 0, 0) || 4 * 32 * kMaxCols > pass_gd_bytes(ng)) return false;
    return true;
}
static_assert(scratch_fits(), "at every NG rankk's arrays lie in one warp's scratch, the sequential walk's columns in gd");

template <int N>
struct Const {              // a compile-time number as an argument
    static constexpr int value = N;
};

// Pass counts of one work item on one warp (lane 0's are used), two 16-bit
// counts to a word: an item has fewer than 2^16 passes
struct Diag {
    unsigned sort_tie, block_exact, irregular;
};

template <int NE>
struct ColSum {
    float T, add, e[NE];
};

// A column's value on element (i, j) is u(i) + v(j) (T: dk1(i) [a1] + dk2(j) a2;
// earlier gas: its column at i; added gas: k2(j)); acc += sw * value, sw the
// element's weight (times its share).  Whole warp.
template <int NE>
__device__ __forceinline__ void add_columns(ColSum<NE>& acc, unsigned w, float sw, float uT, const float* uE, float vT,
                                            float vAdd) {
    const int i = w >> 5;
    const float t = __shfl_sync(kFull, uT, i) + __shfl_sync(kFull, vT, w);
    acc.T = fmaf(sw, t, acc.T);
    acc.add = fmaf(sw, __shfl_sync(kFull, vAdd, w), acc.add);
#pragma unroll
    for (int e = 0; e < NE; ++e) acc.e[e] = fmaf(sw, __shfl_sync(kFull, uE[e], i), acc.e[e]);
}

// The bins of one pass, lane b bin b (rankg.f:118-146).  k: the split
// remainder, the whole elements and the split fraction in the sorted order,
// every operation rounded as in the reference, then / sngl(sum); the gradient
// columns (they feed only the Jacobian, so any order is allowed) in the same
// walk.  The walk runs as long as the longest bin; a lane whose bin has ended
// adds the pad.  The sum of a bin's weights needs no walk: it is a difference
// of the exact prefix, rounded once more or less than the reference's running
// sum, and where that could move its REAL value (the sum within 2^-43 of a
// rounding boundary) the running sum is formed as well.
template <int NE>
__device__ __forceinline__ void walk_bins(const PassScratch& ps, int ng, int nloop, int empty, int lane, int c_last, int sp, double frac, double gprev, double tot, float ws, unsigned word, float a,
                                          float b, float dg, float uT, int nE, float vT, float vAdd, float& kg, float& cT,
                                          float& cAdd) {
    const bool opens = lane > 0 && lane < ng && lane <= c_last, closes = lane < c_last;
    // the split element of the boundary below the bin
    const double f0 = __shfl_up_sync(kFull, frac, 1), g0 = __shfl_up_sync(kFull, gprev, 1);
    const float w0 = __shfl_up_sync(kFull, ws, 1);
    const unsigned word0 = __shfl_up_sync(kFull, word, 1);
    const int sp0 = __shfl_up_sync(kFull, sp, 1);
    const bool in = lane < ng && lane <= c_last;
    const int p0 = opens ? sp0 + 1 : 0, pend = closes ? sp : nloop;
    const int cnt = in ? pend - p0 : 0;
    float uE[NE];
#pragma unroll
    for (int e = 0; e < NE; ++e) uE[e] = e < nE && lane < ng ? ps.col[e * ng + lane] : 0.0f;
    ColSum<NE> g;
    g.T = 0.0f;
    g.add = 0.0f;
#pragma unroll
    for (int e = 0; e < NE; ++e) g.e[e] = 0.0f;
    // keys of the two split elements
    const float key0 = __fadd_rn(__shfl_sync(kFull, a, word0 >> 5), __shfl_sync(kFull, b, word0));
    const float key1 = __fadd_rn(__shfl_sync(kFull, a, word >> 5), __shfl_sync(kFull, b, word));
    const float sr = opens ? __double2float_rn(__dsub_rn(1.0, f0)) : 0.0f;
    const float sf = closes ? __double2float_rn(frac) : 0.0f;
    float acc = opens ? __fmul_rn(__fmul_rn(sr, key0), w0) : 0.0f;
    add_columns<NE>(g, opens ? word0 : kIdMask, opens ? __fmul_rn(sr, w0) : 0.0f, uT, uE, vT, vAdd);
    const int nmax = __reduce_max_sync(kFull, cnt);
#pragma unroll 1
    for (int k = 0; k < nmax; ++k) {
        const uint2 r = ps.rec[k < cnt ? p0 + k : empty];
        const float w = __fmul_rn(__shfl_sync(kFull, dg, r.y >> 5), __shfl_sync(kFull, dg, r.y));
        acc = __fadd_rn(acc, __uint_as_float(r.x));
        add_columns<NE>(g, r.y, w, uT, uE, vT, vAdd);
    }
    if (closes) acc = __fadd_rn(acc, __fmul_rn(__fmul_rn(sf, key1), ws));
    add_columns<NE>(g, closes ? word : kIdMask, closes ? __fmul_rn(sf, ws) : 0.0f, uT, uE, vT, vAdd);
    // the normalisation: sngl(sum of the bin's weights)
    const double first = opens ? __dmul_rn(__dsub_rn(1.0, f0), (double)w0) : 0.0;
    const double whole = __dsub_rn(closes ? gprev : tot, opens ? __dadd_rn(g0, (double)w0) : 0.0);
    const double last = closes ? __dmul_rn(frac, (double)ws) : 0.0;
    double sum = __dadd_rn(__dadd_rn(first, whole), last);
    float nf = __double2float_rn(sum);
    const bool unsure = in && __double2float_rn(sum * (1.0 - 0x1p-43)) != __double2float_rn(sum * (1.0 + 0x1p-43));
    if (__any_sync(kFull, unsure)) {
        sum = first;
#pragma unroll 1
        for (int k = 0; k < nmax; ++k) {
            const unsigned q = ps.rec[k < cnt ? p0 + k : empty].y;
            sum = __dadd_rn(sum, (double)__fmul_rn(__shfl_sync(kFull, dg, q >> 5), __shfl_sync(kFull, dg, q)));
        }
        sum = __dadd_rn(sum, last);
        nf = __double2float_rn(sum);
    }
    if (!closes && lane != ng - 1) nf = 1.0f;   // the last bin reached, left open
    kg = in ? (closes || lane == ng - 1 ? __fdiv_rn(acc, nf) : acc) : 0.0f;
    const float inv = in && nf != 0.0f ? __frcp_rn(nf) : 0.0f;
    cT = quotient(g.T, nf, inv);
    cAdd = quotient(g.add, nf, inv);
#pragma unroll
    for (int e = 0; e < NE; ++e)
        if (e < nE && lane < ng) ps.col[e * ng + lane] = quotient(g.e[e], nf, inv);
}

// One overlap pass.  On entry lane g holds a = k1(g) [* a1], b = k2(g) * a2, the
// T column uT and (in ps.col) the nE gas columns of the distribution so far, the
// added gas's vT = dk2(g) * a2 and vAdd = k2(g), and dg = delg(g) (all zero on
// lanes >= ng), gb = g_ord(g + 1).  mono: k2 is monotone in g and the amounts
// are not negative.  On exit kg, uT, ps.col and cAdd (the added gas's column) hold
// the new distribution.  NGC: NG as a compile-time constant, or 0.
//
// The words leave out the low bits of the keys, so two elements whose keys
// differ only there may come out in the wrong order; the exact keys of every
// neighbouring pair are compared, and if one is wrong (0.3 % of the passes of
// the synthetic configurations) the rows are merged once more on words made of
// the first position of each group of equal leading bits and the low bits,
// which order the elements exactly, equal keys by element.
template <int E, int NGC>
__device__ __forceinline__ void sort_pass(const BatchDev& B, const PassScratch& ps, int ng_run, bool mono, float a, float b,
                                          float dg, double gb, float& uT, int nE, float vT, float vAdd, float& kg,
                                          float& cAdd, int lane, Diag& dgn, int dbg_rec) {
    const int ng = NGC ? NGC : ng_run, nloop = NGC ? NGC * NGC : ng_run * ng_run;
    const float kMax = 3.402823466e38f;
    constexpr unsigned kTop = (E ? kPad : kEnd) >> kIdBits;   // leading bits stay below
    constexpr int kBits = E ? 21 : 22;
    float x[E ? E : 1];
    bool exact = false, disjoint = false;
    // the smallest key's bits, and how many low bits of key - smallest key the words leave out
    auto key_range = [&](unsigned& smin, int& sh) {
        const unsigned abits = __float_as_uint(a);
        const float amin = __uint_as_float(__reduce_min_sync(kFull, lane < ng ? abits : kFull));
        const float amax = __uint_as_float(__reduce_max_sync(kFull, lane < ng ? abits : 0u));
        smin = __float_as_uint(__fadd_rn(amin, __shfl_sync(kFull, b, 0)));
        const unsigned range = __float_as_uint(__fadd_rn(amax, __shfl_sync(kFull, b, ng - 1))) - smin;
        sh = max(0, 32 - __clz(range) - kBits);
        if ((range >> sh) >= kTop) ++sh;
    };
    // ---- words -------------------------------------------------------------
    // inputs not monotone in g, negative, infinite or NaN, and keys spread over
    // more than 31 bits, take the reference heapsort
    bool net = mono && __all_sync(kFull, a >= 0.0f && a <= kMax && b >= 0.0f && b <= kMax);
    int sh = 0;
    unsigned smin = 0;
    if (net) {
        a = __fadd_rn(a, 0.0f);                  // -0 -> +0
        key_range(smin, sh);
        net = sh <= (int)kIdBits;
        // every row's keys lie at or above those of the row before: the elements are in order as they are
        const float an = __shfl_down_sync(kFull, a, 1);
        const float b0 = __shfl_sync(kFull, b, 0), bl = __shfl_sync(kFull, b, ng - 1);
        disjoint = __all_sync(kFull, lane + 1 >= ng || __fadd_rn(an, b0) >= __fadd_rn(a, bl));
        disjoint = disjoint && net;
        dgn.block_exact += disjoint;
    }
    const int ch = (nloop + 31) >> 5;            // sorted positions a lane runs over below, pads at the end
    const int c0 = lane * ch;
    if (lane >= ng) a = __int_as_float(0x7fffffff);   // a pad's key: NaN, neither below nor equal to any
    unsigned* gw = (unsigned*)ps.gd;
    unsigned* rw = (unsigned*)ps.rec;
    int levels = 0;
    while ((ng << levels) < nloop) ++levels;
    unsigned* rows = (levels & 1) ? gw : rw;     // where the merge reads the rows
    if (disjoint) {
#pragma unroll 1
        for (int p = lane; p < 32 * ch; p += 32) {
            const int i = p / ng;
            ps.rec[p].y = p < nloop ? (unsigned)(i << 5 | (p - i * ng)) : kIdMask;
        }
    } else if (net) {
        const unsigned mul = 1u << (kIdBits - sh), sub = smin * mul;
        if (E) {
            int i = lane / ng, j = lane - i * ng;
            const int di = 32 / ng, dj = 32 - di * ng;
#pragma unroll
            for (int t = 0; t < E; ++t) {
                const unsigned kb = __float_as_uint(__fadd_rn(__shfl_sync(kFull, a, i), __shfl_sync(kFull, b, j)));
                x[t] = __uint_as_float(t * 32 + lane < nloop ? ((kb * mul - sub) & ~kIdMask) | (unsigned)(i << 5 | j) : kPad);
                j += dj;
                i += di;
                if (j >= ng) {
                    j -= ng;
                    ++i;
                }
            }
        } else {
#pragma unroll 4
            for (int i = 0; i < ng; ++i) {
                const unsigned kb = __float_as_uint(__fadd_rn(__shfl_sync(kFull, a, i), b));
                if (lane <= ng)
                    rows[i * (ng + 1) + lane] = lane < ng ? ((kb * mul - sub) & ~kIdMask) | (unsigned)(i << 5 | lane) : kEnd;
            }
        }
    }
    // the reference heapsort on the elements in nloop order (sort2g.f); its
    // words live in gd
    auto heapsort_pass = [&]() {
        __syncwarp();
        unsigned long long* W = (unsigned long long*)ps.gd;
#pragma unroll 1
        for (int e = lane; e - lane < nloop; e += 32) {
            const int i = min(e / ng, 31), j = e - (e / ng) * ng;
            const float key = __fadd_rn(__shfl_sync(kFull, a, i), __shfl_sync(kFull, b, j));
            if (e < nloop) W[e] = ((unsigned long long)__float_as_uint(key) << 32) | (unsigned)e;
        }
        __syncwarp();
        if (lane == 0) heapsort_words(nloop, W);
        __syncwarp();
#pragma unroll 1
        for (int p = lane; p < 32 * ch; p += 32) {
            const int e = p < nloop ? (int)(unsigned)W[p] : 0, i = e / ng;
            ps.rec[p].y = p < nloop ? (unsigned)(i << 5 | (e - i * ng)) : kIdMask;
        }
        __syncwarp();
        exact = true;
        dgn.block_exact += 0x10000u;
    };
    if (!net) heapsort_pass();

    // ---- sort, cumulative weights, bin boundaries, tie checks ----------------
    // Each lane runs over a chunk of consecutive sorted positions: the FP64
    // prefix of the weights (every partial sum is exact, so any order gives the
    // reference's values) and the exact keys of neighbours; a warp scan of the
    // lanes' totals; then lane b finds boundary b (the first position whose
    // cumulative weight reaches g_ord(b+1), rankg.f:119-129) and its split
    // fraction.
    bool again = false, counted = false;
    int sp, c_last;
    double frac, gprev, tot;
    float ws;
    unsigned word;
    bool irregular, gerr;
    for (;;) {
        __syncwarp();
        if (!exact && !disjoint) {
            if (E) {
                // through gd, position p at p + (p >> 4): lanes writing E consecutive positions do not share a bank
                warp_sort<E ? E : 1>(x, lane);
#pragma unroll
                for (int t = 0; t < E; ++t)
                    if (lane * E + t < nloop) gw[lane * E + ((lane * E) >> 4) + t] = __float_as_uint(x[t]);
                __syncwarp();
                for (int p = lane; p < nloop; p += 32) ps.rec[p].y = gw[p + (p >> 4)];
            } else {
                merge_rows<NGC>((unsigned)__cvta_generic_to_shared(gw), (unsigned)__cvta_generic_to_shared(rw), ps.mtab, ng,
                                levels, lane);
            }
            for (int p = nloop + lane; p < 32 * ch; p += 32) ps.rec[p].y = kIdMask;
            __syncwarp();
        }
        double run = 0.0;
        bool wrong = false, tie = false;
        const unsigned qprev = lane > 0 ? ps.rec[c0 - 1].y : kIdMask;   // lane 0: a pad
        float kprev = __fadd_rn(__shfl_sync(kFull, a, qprev >> 5), __shfl_sync(kFull, b, qprev));
#pragma unroll 1
        for (int p = c0; p < c0 + ch; ++p) {
            const unsigned q = ps.rec[p].y;
            const float key = __fadd_rn(__shfl_sync(kFull, a, q >> 5), __shfl_sync(kFull, b, q));
            const float w = __fmul_rn(__shfl_sync(kFull, dg, q >> 5), __shfl_sync(kFull, dg, q));
            run = __dadd_rn(run, (double)w);
            ps.gd[p] = run;
            ps.rec[p].x = __float_as_uint(__fmul_rn(key, w));
            wrong |= key < kprev;
            tie |= key == kprev;
            kprev = key;
        }
        if (lane == 0) ps.rec[32 * ch] = make_uint2(0u, kIdMask);
        if (!exact && !disjoint && !again && __any_sync(kFull, wrong)) {
            // words anew: the first position of the element's group of equal
            // leading bits << sh | the bits left out so far
            unsigned sm;
            int sb;
            key_range(sm, sb);
            auto starts = [&](int p, unsigned q) { return p == 0 || ((ps.rec[p - 1].y ^ q) >> kIdBits) != 0; };
            int first = 0;
#pragma unroll 1
            for (int p = c0; p < min(c0 + ch, nloop); ++p)
                if (starts(p, ps.rec[p].y)) first = p;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) first = max(first, __shfl_up_sync(kFull, first, o));
            first = __shfl_up_sync(kFull, first, 1);   // of the position before the chunk (lane 0 starts a group)
            // the new words go to gd, in their rows' order for the merge
            __syncwarp();
#pragma unroll 1
            for (int p = c0; p < c0 + ch; ++p) {
                const bool live = p < nloop;
                const unsigned q = ps.rec[p].y;
                const float key = __fadd_rn(__shfl_sync(kFull, a, q >> 5), __shfl_sync(kFull, b, q));
                if (live) {
                    if (starts(p, q)) first = p;
                    const unsigned rest = (__float_as_uint(key) - sm) & ((1u << sb) - 1);
                    const unsigned w = ((((unsigned)first << sb) | rest) << kIdBits) | (q & kIdMask);
                    gw[E ? p : ((q >> 5) & 31) * (ng + 1) + (q & 31)] = w;
                }
            }
            __syncwarp();
            if (E) {
#pragma unroll
                for (int t = 0; t < E; ++t) x[t] = __uint_as_float(lane * E + t < nloop ? gw[lane * E + t] : kPad);
            } else {
                if (lane < ng) gw[lane * (ng + 1) + ng] = kEnd;
                if (rows != gw) {
                    __syncwarp();
                    for (int p = lane; p < ng * (ng + 1); p += 32) rw[p] = gw[p];
                }
            }
            again = true;
            continue;
        }
        double incl = run;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double t = __shfl_up_sync(kFull, incl, o);
            if (lane >= o) incl = __dadd_rn(incl, t);
        }
        const double base = __dsub_rn(incl, run);   // exact: every partial sum is exact
        __syncwarp();
        // boundary b = lane: the lane L whose positions the prefix reaches gb in
        // (a search over the lanes' totals), then the position t of that lane
        int L = 0;
#pragma unroll
        for (int st = 16; st >= 1; st >>= 1) {
            const double v = __shfl_sync(kFull, incl, L + st - 1);
            if (v < gb) L += st;
        }
        tot = __shfl_sync(kFull, incl, 31);
        const double bL = __shfl_sync(kFull, base, L);
        const int lo0 = L * ch;
        const bool found = lane < ng && tot >= gb;
        sp = nloop;
        if (found) {
            int lo = lo0, hi = lo0 + ch;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (__dadd_rn(ps.gd[mid], bL) >= gb) hi = mid; else lo = mid + 1;
            }
            sp = lo;
        }
        gprev = sp < nloop && sp > lo0 ? __dadd_rn(ps.gd[sp - 1], bL) : bL;
        word = sp < nloop ? ps.rec[sp].y : kIdMask;
        ws = __fmul_rn(__shfl_sync(kFull, dg, word >> 5), __shfl_sync(kFull, dg, word));
        frac = sp < nloop ? __ddiv_rn(__dsub_rn(gb, gprev), (double)ws) : 0.0;
        // one element crossing two boundaries: equal split positions
        const int sp_next = __shfl_down_sync(kFull, sp, 1);
        irregular = __any_sync(kFull, lane + 1 < ng && sp < nloop && sp == sp_next);
        c_last = __popc(__ballot_sync(kFull, sp < nloop));
        const int sp_last = __shfl_sync(kFull, sp, ng - 1);
        gerr = c_last == ng && sp_last < nloop - 1;    // elements left after the last boundary
        const bool anytie = __any_sync(kFull, tie);
        if (!counted) {
            dgn.sort_tie += anytie ? 0x10001u : 1u;
            counted = true;
        }
        if (exact || !anytie) break;
        // a split element whose key equals a neighbour's: the tie order decides the bins
        bool risky = B.strict_ties != 0;
        if (!risky) {
            const unsigned qn = sp + 1 < nloop ? ps.rec[sp + 1].y : kIdMask;
            const unsigned qp = sp < nloop && sp > 0 ? ps.rec[sp - 1].y : kIdMask;
            const float kc = __fadd_rn(__shfl_sync(kFull, a, word >> 5), __shfl_sync(kFull, b, word));
            const float kn = __fadd_rn(__shfl_sync(kFull, a, qn >> 5), __shfl_sync(kFull, b, qn));
            const float kp = __fadd_rn(__shfl_sync(kFull, a, qp >> 5), __shfl_sync(kFull, b, qp));
            risky = __any_sync(kFull, sp < nloop && ((sp > 0 && kp == kc) || (sp + 1 < nloop && kn == kc)));
        }
        if (!risky) break;
        heapsort_pass();
    }
    if (gerr) atomicOr(B.status, kStGord);
    int16_t* dbg_split = nullptr;
    if (dbg_rec >= 0) {
        int16_t* dbg_perm = B.dbg_perm + (int64_t)dbg_rec * nloop;
        dbg_split = B.dbg_split + (int64_t)dbg_rec * ng;
#pragma unroll 1
        for (int p = lane; p < nloop; p += 32) {
            const unsigned q = ps.rec[p].y;
            dbg_perm[p] = (int16_t)(((q >> 5) & 31) * ng + (q & 31));
        }
        if (lane < ng) dbg_split[lane] = (int16_t)(!irregular && sp < nloop ? sp : -1);
        __syncwarp();
    }
    if (irregular) {
        // sequential rankg walk (rankg.f:118-152): every lane follows it, the
        // lane of the current bin accumulates
        dgn.irregular += 1;
        float acc = 0.0f, nT = 0.0f, nA = 0.0f;
        float* nc = (float*)ps.gd;               // the gas columns' new values
        for (int c = 0; c < nE; ++c) nc[c * 32 + lane] = 0.0f;   // lanes' own entries
        int ig = 0;
        double sum = 0.0, gp = 0.0;
#pragma unroll 1
        for (int p = 0; p < nloop; ++p) {
            const unsigned q = ps.rec[p].y;
            const float key = __fadd_rn(__shfl_sync(kFull, a, q >> 5), __shfl_sync(kFull, b, q));
            const float w = __fmul_rn(__shfl_sync(kFull, dg, q >> 5), __shfl_sync(kFull, dg, q));
            const double gcur = __dadd_rn(gp, (double)w);
            if (ig >= ng) {
                if (lane == 0) atomicOr(B.status, kStGord);
                break;
            }
            const double go = __shfl_sync(kFull, gb, ig);
            const bool closes = !(gcur < go);
            const double fr = closes ? __ddiv_rn(__dsub_rn(go, gp), __dsub_rn(gcur, gp)) : 1.0;
            float share = closes ? __double2float_rn(fr) : 1.0f;
            const float tv = __fadd_rn(__shfl_sync(kFull, uT, q >> 5), __shfl_sync(kFull, vT, q));
            const float av = __shfl_sync(kFull, vAdd, q);
#pragma unroll 1
            for (int part = 0; part < 2; ++part) {
                // part 0: the element's share of bin ig; part 1 (a split element): the rest to the next bin
                if (lane == ig) {
                    acc = __fadd_rn(acc, __fmul_rn(__fmul_rn(share, key), w));
                    nT = __fadd_rn(nT, __fmul_rn(__fmul_rn(share, tv), w));
                    nA = __fadd_rn(nA, __fmul_rn(__fmul_rn(share, av), w));
                }
                if (lane == ig)
                    for (int c = 0; c < nE; ++c)
                        nc[c * 32 + lane] = __fadd_rn(nc[c * 32 + lane],
                                                      __fmul_rn(__fmul_rn(share, ps.col[c * ng + ((q >> 5) & 31)]), w));
                if (part == 0) {
                    sum = closes ? __dadd_rn(sum, __dmul_rn(fr, (double)w)) : __dadd_rn(sum, (double)w);
                    if (!closes) break;
                    const float fs = __double2float_rn(sum);
                    if (lane == ig) {
                        acc = __fdiv_rn(acc, fs);
                        nT = __fdiv_rn(nT, fs);
                        nA = __fdiv_rn(nA, fs);
                        for (int c = 0; c < nE; ++c) nc[c * 32 + lane] = __fdiv_rn(nc[c * 32 + lane], fs);
                    }
                    if (dbg_split && lane == 0) dbg_split[ig] = (int16_t)p;
                    ig = ig + 1;
                    sum = __dmul_rn(__dsub_rn(1.0, fr), (double)w);
                    share = __double2float_rn(__dsub_rn(1.0, fr));
                    if (ig >= ng) break;
                }
            }
            gp = gcur;
        }
        if (ig == ng - 1 && lane == ig) {
            const float fs = __double2float_rn(sum);
            acc = __fdiv_rn(acc, fs);
            nT = __fdiv_rn(nT, fs);
            nA = __fdiv_rn(nA, fs);
            for (int c = 0; c < nE; ++c) nc[c * 32 + lane] = __fdiv_rn(nc[c * 32 + lane], fs);
        }
        kg = acc;
        uT = nT;
        cAdd = nA;
        __syncwarp();
        if (lane < ng)
            for (int c = 0; c < nE; ++c) ps.col[c * ng + lane] = nc[c * 32 + lane];
        __syncwarp();
        return;
    }

    // ---- k(g) and gradient columns -------------------------------------------
    // specialised on the number of gas columns that are not zero before the pass
    float cT;
    auto walk = [&](auto n) {
        walk_bins<decltype(n)::value>(ps, ng, nloop, 32 * ch, lane, c_last, sp, frac, gprev, tot, ws, word, a, b, dg, uT, nE,
                                      vT, vAdd, kg, cT, cAdd);
    };
    if (nE <= 1) walk(Const<1>());
    else if (nE == 2) walk(Const<2>());
    else if (nE == 3) walk(Const<3>());
    else walk(Const<kMaxCols>());
    uT = cT;
    __syncwarp();
}

}  // namespace rtb
