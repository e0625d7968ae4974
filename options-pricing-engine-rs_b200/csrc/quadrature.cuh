// Warp-cooperative greedy globally-adaptive Gauss-Kronrod-15 on [0, 1].
//
// Reference: heston.rs:180-212 (gk15_panel, adaptive_gk), heston.rs:29-59
// (nodes/weights), heston.rs:220-229 (gk_integrate).
//
// One warp integrates one integral.  Each step bisects the live panel with
// the largest error estimate: lanes 0-14 evaluate the 15 Kronrod nodes of the
// left child and lanes 16-30 those of the right child (30 of 32 lanes busy);
// a half-warp reduce-scatter forms the K15 and G7 sums.  The live-panel list
// (at most 200 entries of {err, K, a, b}) sits in shared memory, one list per
// warp, and is maintained exactly as the reference maintains its Vec:
//   * argmax by f64::total_cmp with the LAST maximum winning ties (errors are
//     non-negative, so their IEEE bit patterns compare as unsigned integers
//     in total_cmp order, and so do their leading bits);
//   * swap_remove of the chosen panel, then push(left), push(right);
//   * total += kl + kr - kw; err += el + er - ew, in that association;
//   * stop when err <= tol or 200 panels are live.
// Node positions c + h*x_i and the panel products K*h, |K-G|*h are rounded
// exactly as the reference rounds them (no FMA contraction), so the panel
// geometry is bit-identical; only the integrand values and the order of the
// 15-term sums differ at the last-ulp level.
#pragma once

#include "cf_device.cuh"
#include "checked.cuh"

namespace ope {

constexpr int kMaxPanels = 200;  // heston.rs:194

// GK15 nodes and weights in the reference's order (heston.rs:29-49) with a
// zero pad at index 15, and the G7 weight scattered onto its Kronrod index
// (G7_IDX = {0,3,4,7,8,11,12}, heston.rs:53-59), zero elsewhere.
static __constant__ double c_gk_x[16] = {
    0.0,
    0.2077849550078985, -0.2077849550078985,
    0.4058451513773972, -0.4058451513773972,
    0.5860872354676911, -0.5860872354676911,
    0.7415311855993945, -0.7415311855993945,
    0.8648644233597691, -0.8648644233597691,
    0.9491079123427585, -0.9491079123427585,
    0.9914553711208126, -0.9914553711208126,
    0.0};
static __constant__ double c_gk_wk[16] = {
    0.2094821410847278,
    0.2044329400752989, 0.2044329400752989,
    0.1903505780647854, 0.1903505780647854,
    0.1690047266392679, 0.1690047266392679,
    0.1406532597155259, 0.1406532597155259,
    0.1047900103222502, 0.1047900103222502,
    0.0630920926299786, 0.0630920926299786,
    0.0229353220105292, 0.0229353220105292,
    0.0};
static __constant__ double c_gk_wg[16] = {
    0.4179591836734694,
    0.0, 0.0,
    0.3818300505051189, 0.3818300505051189,
    0.0, 0.0,
    0.2797053914892766, 0.2797053914892766,
    0.0, 0.0,
    0.1294849661688697, 0.1294849661688697,
    0.0, 0.0,
    0.0};

// One warp's live-panel list (structure of arrays, 6400 bytes).
struct alignas(16) PanelStore {
    unsigned long long ekey[kMaxPanels];  // error as IEEE bits (total_cmp order for err >= 0)
    double k[kMaxPanels];
    double2 ab[kMaxPanels];
};

// Per-lane quadrature constants, loaded once per warp.
struct LaneRule {
    double x, wk, wg;
    int half;   // 0 = left child, 1 = right child
    // reduce-scatter weights: of the K15 and G7 weights of this lane's node,
    // the one whose product the lane keeps (G7 if lane bit 3 is set) and the
    // one whose product it sends to lane ^ 8
    double wkeep, wsend;
    // word of the panel list's entry 0 this lane moves on a swap_remove
    // (lanes 0-3: ekey, k, a, b), as a byte offset, and that word's stride
    unsigned copy_at, copy_by;
};

__device__ __forceinline__ LaneRule lane_rule(int lane) {
    LaneRule R;
    const int j = lane & 15;
    R.x = c_gk_x[j];
    R.wk = c_gk_wk[j];
    R.wg = c_gk_wg[j];
    R.half = lane >> 4;
    R.wkeep = (lane & 8) ? R.wg : R.wk;
    R.wsend = (lane & 8) ? R.wk : R.wg;
    R.copy_at = lane == 0 ? 0u : 1600u * (unsigned)min(lane, 2) + (lane == 3 ? 8u : 0u);
    R.copy_by = lane < 2 ? 8u : 16u;
    return R;
}

// K15 and G7 sums of each half-warp's child.  A reduce-scatter over the
// half-warp: at the first exchange (lanes i and i^8) the lanes with bit 3
// clear keep a K15 partial sum and those with it set a G7 partial sum (each
// lane sends the product its partner keeps), and three more xor levels
// finish each sum with one shuffle per level.  Every lane adds the same two
// partial sums at each level (commuted in its partner), so all lanes of a
// quarter hold bit-identical totals, summed in the pairing order (8, 4, 2, 1):
// K15 in the lanes with bit 3 clear, G7 in the others.
__device__ __forceinline__ double gk_sums(double f, const LaneRule& R) {
    const unsigned FULL = 0xffffffffu;
    double v = fma(R.wkeep, f, __shfl_xor_sync(FULL, __dmul_rn(R.wsend, f), 8));
    v = __dadd_rn(v, __shfl_xor_sync(FULL, v, 4));
    v = __dadd_rn(v, __shfl_xor_sync(FULL, v, 2));
    return __dadd_rn(v, __shfl_xor_sync(FULL, v, 1));
}

// The run cache: node_cf's values at the panels that the contracts of one
// run (consecutive contracts of one surface with the same expiry and rate,
// integrating the same P1 or P2) have bisected, kept by the one warp that
// integrates the run's contracts one after another.  Every panel of the
// quadrature descends from [0, 1] by bisection and a bisection always
// evaluates both children, so the cached panels form a binary tree: entry 0
// is [0, 1], and each entry records the entries of its two children once
// they have been evaluated.  Each live panel of the running integral carries
// its entry (kNoEntry: not cached, nor are its descendants), so a bisection
// finds its children's values with one load, without searching.  A contract
// whose next panel is in the tree skips node_cf (the CF, its square root,
// logarithm and exponentials) and pays only node_finish (its own phase and
// one sine).  The tree lives in global memory (per warp: cap entries of 15
// nodes x {W, A}); when it is full, further panels are evaluated
// uncached.  The cached values are the ones node_cf's result gives (u is
// recomputed from the node, bit for bit), so a contract's price is
// bit-identical with and without the cache.  An entry is two whole
// 128-byte lines (15 nodes and the pad lane's, so that L2 never fetches the
// rest of a partly written line from DRAM).
constexpr int kRunEntries = 127;    // entries of one run's tree at most
constexpr int kNoEntry = 127;       // not cached; as an entry it has no children
constexpr int kRunLinks = 128;

struct RunCacheWarp {
    double2* wa;     // [cap][16]: W and Im Z without the phase (NodeCf)
    uint8_t* child;  // shared, [kRunLinks]: left child's entry, the right one's is the next (kNoEntry: none yet)
    uint8_t* slot;   // shared, [kMaxPanels]: entry of each live panel of the running integral
    int cap;         // entries (1..kRunEntries)
    int n_alloc;     // entries in use (warp-uniform; 0 at the start of a run)
};

// End of a run: its entries will be rewritten before they are read again, so
// their lines are dropped from L2 without being written back to DRAM
// (discard.global.L2), which keeps the dead data of finished runs from
// costing DRAM bandwidth.  Warp-collective.
__device__ __forceinline__ void run_cache_discard(RunCacheWarp& rc, int lane) {
    __syncwarp();
    for (int j = lane; j < 2 * rc.n_alloc; j += 32)
        asm volatile("discard.global.L2 [%0], 128;" ::"l"(rc.wa + (size_t)j * 8) : "memory");
    __syncwarp();
    rc.n_alloc = 0;
}

// The panel of largest error, the last of equals, by all 64 bits of the keys
// (errors are non-negative, so their bits order as they do).
static __device__ __noinline__ int argmax_exact(const PanelStore& L, int len, int lane) {
    const unsigned FULL = 0xffffffffu;
    unsigned long long best = 0ull;
    int bi = -1;
    for (int i = lane; i < len; i += 32) {
        const unsigned long long kk = L.ekey[i];
        if (kk >= best) { best = kk; bi = i; }
    }
    // high word, then low word among the lanes holding the top high word, then
    // the largest index holding both
    const unsigned hi = (unsigned)(best >> 32), lo = (unsigned)best;
    const unsigned mh = __reduce_max_sync(FULL, hi);
    const unsigned ml = __reduce_max_sync(FULL, hi == mh ? lo : 0u);
    return (int)__reduce_max_sync(FULL, (hi == mh && lo == ml) ? (unsigned)(bi + 1) : 0u) - 1;
}

// Step hooks of gk_integrate_warp.  The pricing kernels use NoTrace (empty
// and inlined: no code); the QAG trace kernel (trace.cu) records every step.
//   first(lane, f, k0, e0): the first panel [0, 1] (f: this lane's integrand
//     value, lanes 0-14 hold the 15 nodes);
//   step(j, lane, f, a, b, ew, k, e, kx, ex, err, total): bisection j of a
//     panel of error estimate ew; [a, b], k and e are this half-warp's child,
//     its K and error estimate, kx and ex the other half's; then the running
//     error and total after it (k, kx, total: in the lanes with bit 3 clear).
struct NoTrace {
    __device__ __forceinline__ void first(int, double, double, double) const {}
    __device__ __forceinline__ void step(int, int, double, double, double, double, double, double, double, double,
                                         double, double) const {}
};

// What bounds a step besides its node: issue slots.  Each half-warp keeps its
// own child's sums and writes its own list entry (one leader lane each), and
// the four words of a swap_remove move in one load and one store; with both
// children's values in every lane and lane 0 writing the whole list, the
// 262k-contract Bates batch took 10.17 ms instead of 9.79, the run kernel's
// 1.46M-contract grids 32.4 ms instead of 27.2.  The argmax on 24 bits of each
// error with its index (one maximum over the warp instead of three, no
// selects), the first step without branches of its own, and the run cache's
// links in shared memory: 9.27 -> 9.05 and 27.0 -> 24.7 ms.
//
// Returns the integral (in the lanes with bit 3 clear).  `nbis` receives the
// number of bisections (loop iterations of heston.rs:200-210); the final
// live-panel list (nbis + 1 entries) is left in L.  The first panel and every
// bisection go through ONE call site of the integrand, so the (large) inlined
// node evaluation exists once in the instruction stream.
//
// CACHED: with the run cache `rc`: each
// step first looks its panel(s) up in the tree (a hit: both children, or the
// root, already evaluated) and otherwise evaluates node_cf and, while the
// tree has room and the bisected panel is in it, stores the children.
template <bool BATES, bool CACHED = false, class Trace = NoTrace>
__device__ __forceinline__ double gk_integrate_warp(const CfConsts& C, double tol, PanelStore& L, int lane,
                                                    const LaneRule& R, int* nbis, const Trace& tr = Trace(),
                                                    RunCacheWarp* rc = nullptr) {
    const unsigned FULL = 0xffffffffu;
    double total = 0.0, err = 0.0;
    int len = 0;
    // panel under evaluation in this half-warp; first step: [0, 1] on the left,
    // an empty panel, which adds nothing, on the right
    double pa = R.half ? 0.5 : 0.0, pb = R.half ? 0.5 : 1.0, kw = 0.0, ew = 0.0;
    char* const list = reinterpret_cast<char*>(&L);
    // errors beyond the live panels read as 0 in the argmax
#pragma unroll
    for (int j = 0; j < (kMaxPanels + 31) / 32; ++j)
        if (lane + 32 * j < kMaxPanels) L.ekey[lane + 32 * j] = 0ull;
    __syncwarp();
    // cache mode of the step (warp-uniform): hit = read entries el_ and el_ + 1,
    // put = evaluate and store into them; neither = evaluate uncached.  The
    // first step's panel [0, 1] is entry 0.
    bool hit = false, put = false;
    int el_ = 0, sw_ = kNoEntry;  // left child's entry (the right one's is the next), entry of the bisected panel
    if (CACHED) {
        hit = rc->n_alloc > 0;
        put = !hit;
        if (put) rc->n_alloc = 1;
    }
    while (true) {
        const double c = 0.5 * (pa + pb), h = 0.5 * (pb - pa);
        const double tn = __dadd_rn(c, __dmul_rn(h, R.x));
        // the node's strike-free part: W, A, u (from the tree on a hit).  The
        // pad lanes 15 and 31 evaluate the panel's centre; their weights are 0.
        double nw, na, nu;
        if (CACHED && hit) {
            // (the first step's right half reads the root's entry too)
            const double2 wa = __ldcg(rc->wa + (el_ + (len > 0 ? R.half : 0)) * 16 + (lane & 15));
            nw = wa.x;
            na = wa.y;
            nu = node_u_of(tn);
        } else {
            const NodeCf nc = node_cf<BATES>(C, tn);
            nw = nc.w;
            na = nc.a;
            nu = nc.u;
            // each half-warp writes its child's entry whole, pad lane included
            if (CACHED && put && (len > 0 || R.half == 0))
                __stcg(rc->wa + (el_ + R.half) * 16 + (lane & 15), make_double2(nw, na));
        }
        const double f = node_finish(C.x, nu, na, nw);
        // K (in the lanes with bit 3 clear) and error of this half's child,
        // then both children's sums
        const double v = gk_sums(f, R);
        const double e = __dmul_rn(fabs(__dsub_rn(v, __shfl_xor_sync(FULL, v, 8))), h), k = __dmul_rn(v, h);
        const double ex = __shfl_xor_sync(FULL, e, 16), kx = __shfl_xor_sync(FULL, k, 16);
        total = __dadd_rn(total, __dsub_rn(__dadd_rn(k, kx), kw));
        err = __dadd_rn(err, __dsub_rn(__dadd_rn(e, ex), ew));
        if (len == 0) {
            tr.first(lane, R.half ? 0.0 : f, k, e);
        } else {
            tr.step(len, lane, f, pa, pb, ew, k, e, kx, ex, err, total);
        }
        // push(left) over the list's last slot (its panel was bisected, or
        // moved to the bisected one's slot below), push(right) behind it (the
        // first step's empty right panel is overwritten by the second's)
        if ((lane & 15) == 0) {
            const int at = max(len - 1, 0) + R.half;
            L.ekey[at] = (unsigned long long)__double_as_longlong(e);
            L.k[at] = k;
            L.ab[at] = make_double2(pa, pb);
            if (CACHED) {
                // the children's entries, with no children of their own yet
                // (a first step's right half leaves the root's alone)
                const int own = el_ == kNoEntry ? kNoEntry : el_ + R.half;
                rc->slot[at] = (uint8_t)own;
                if (put && (len > 0 || R.half == 0)) rc->child[own] = (uint8_t)kNoEntry;
                if (put && len > 0 && R.half == 0) rc->child[sw_] = (uint8_t)el_;
            }
        }
        ++len;
        __syncwarp();
        if (!(err > tol && len < kMaxPanels)) break;
        if (!ope_check(len < kMaxPanels, CHK_PANEL_COUNT)) break;
        // argmax over the live list, last maximum wins (Iterator::max_by): the
        // top 24 bits of each error (exponent and 13 bits; no sign) with its
        // index below them, the largest two per lane over chunks of 32
        // entries (stopping, warp-uniformly, after the last one in use), one
        // warp maximum.  Only where another error shares the winner's 24 bits
        // (vote) are the full 64 bits compared.
        int bi;
        {
            const unsigned* hi = reinterpret_cast<const unsigned*>(L.ekey) + 1;  // high words, 2 apart
            unsigned best = ((hi[2 * lane] << 1) & ~255u) | (unsigned)lane, second = 0u;
#pragma unroll
            for (int j = 1; j < (kMaxPanels + 31) / 32; ++j) {
                if (32 * j >= len) break;
                if (32 * j + 31 < kMaxPanels || lane + 32 * j < kMaxPanels) {
                    const unsigned p = ((hi[2 * lane + 64 * j] << 1) & ~255u) | (unsigned)(lane + 32 * j);
                    second = max(second, min(best, p));
                    best = max(best, p);
                }
            }
            const unsigned top = __reduce_max_sync(FULL, best);
            bi = (int)(top & 255u);
            if (__any_sync(FULL, ((best == top ? second : best) ^ top) < 256u)) bi = argmax_exact(L, len, lane);
        }
        if (!ope_check(bi >= 0 && bi < len, CHK_PANEL_INDEX)) bi = 0;
        const int w = bi, last = len - 1;
        ew = __longlong_as_double((long long)L.ekey[w]);
        kw = L.k[w];
        const double2 ab = L.ab[w];
        const double m = 0.5 * (ab.x + ab.y);
        pa = R.half ? m : ab.x;
        pb = R.half ? ab.y : m;
        unsigned long long word = 0;
        if (lane < 4) word = *reinterpret_cast<const unsigned long long*>(list + (R.copy_at + last * R.copy_by));
        int moved = 0;
        if (CACHED) {
            // the children of panel w: in the tree (hit), or new entries (put)
            // while the tree has room for both and w is in it
            sw_ = rc->slot[w];
            moved = rc->slot[last];
            if (!ope_check(sw_ < rc->n_alloc || sw_ == kNoEntry, CHK_RUN_ENTRY)) sw_ = kNoEntry;
            el_ = rc->child[sw_];
            hit = el_ != kNoEntry;
            if (!ope_check(!hit || el_ + 1 < rc->n_alloc, CHK_RUN_ENTRY)) {
                hit = false;  // evaluate uncached
                el_ = sw_ = kNoEntry;
            }
            put = !hit && sw_ != kNoEntry && rc->n_alloc + 2 <= rc->cap;
            if (put) {
                el_ = rc->n_alloc;
                rc->n_alloc += 2;
            }
        }
        __syncwarp();  // every lane has read entry w before it is overwritten
        // swap_remove: the last entry takes the bisected one's slot (its own: stays,
        // as the left child, written by one lane above, is the next into it)
        if (lane < 4 && w != last) *reinterpret_cast<unsigned long long*>(list + (R.copy_at + w * R.copy_by)) = word;
        if (CACHED && lane == 0) rc->slot[w] = (uint8_t)moved;
    }
    *nbis = len - 1;
    return total;
}

// heston.rs:95-98 + heston.rs:70 (bates.rs:60-62, 37): the Gil-Pelaez
// combination, the max(.,0) clamp on the call, put by parity.  Rounded in the
// reference's association order (no FMA).
__device__ __forceinline__ double finish_price(double s, double k, double t, double r, double q, int opt_type,
                                               double i1, double i2) {
    const double PI = 3.14159265358979323846;
    const double p1 = __dadd_rn(0.5, i1 / PI);
    const double p2 = __dadd_rn(0.5, i2 / PI);
    const double seq = __dmul_rn(s, exp(-q * t));
    const double ker = __dmul_rn(k, exp(-r * t));
    const double call = fmax(__dsub_rn(__dmul_rn(seq, p1), __dmul_rn(ker, p2)), 0.0);
    if (opt_type == 0) return call;
    return __dadd_rn(__dsub_rn(call, seq), ker);
}

}  // namespace ope
