// Fused EM iteration: E-step, statistics reduction and M-step in one
// persistent kernel launch per iteration.
//
// Work: a queue of session tiles (host-built, see model.cu).  Each tile is a
// run of whole queries (or a chunk of one large query) whose qd indices form
// one contiguous window.  The warps of a CTA work in groups, each with its own
// part of shared memory, which holds one tile at a time: the window's values,
// its 16-bit click counts and a bin per private statistic and qd.  A group
// takes a tile at a time:
//   * asynchronous copies (cp.async, completion on an mbarrier) of the window's
//     values and counts into the group's memory.  The descriptor of the next
//     tile is in registers by then, and its data is asked into L2 (bulk copies
//     and bulk prefetches by one thread took longer than the warps' own
//     copies: 0.219 against 0.208 ms when tried);
//   * E-step: chunks of 32 sessions, one session per thread, from the warp's
//     chunk buffer (the next chunk is copied meanwhile), values from the
//     group's memory; each private statistic is added into the bin of its qd,
//     each public one into registers;
//   * M-step:
//       - owned tile (whole queries): four qd per lane, straight from the bins,
//         the old values and the click counts, written in place to global
//         memory (no other tile reads those parameters);
//       - split tile (part of a large query): the group folds the bins into the
//         query's FP64 global bins, and the one that completes the query's last
//         tile runs its M-step.
// The tiles are cut from blocks of up to 1024 packed sessions and 1536 qd (the
// shape's), which set the scale of the fixed-point bins: what a pair's bins add
// up to does not depend on the cut.
// A group is one warp for windows of up to a few hundred qd (narrow tiles):
// then nothing in the loop waits for another warp, and the 24 warps of an SM
// hide each other's copies and recursions.  Measured per iteration at 16M DBN
// sessions: 0.351 ms with a CTA of eight warps per tile and a barrier per tile,
// 0.196 ms with a warp per tile (CCM: 0.387 and 0.217 ms; 1.6M DBN sessions:
// 52 and 41 us).  Three tiles in flight per CTA with counted hand-offs instead
// of the barrier came to 0.236 ms, 0.145 ms of it with the E- and M-steps left
// out: hand-offs and refills.  Wider windows, direct tiles, and queries that would
// be cut at a greater cost (cut_tiles, model.cu) take a whole CTA: up to a block's
// queries a tile, since a tile costs three barriers (one query each: 20,000
// queries of 100 sessions and 500 pairs 209 us per iteration, runs 103, a CTA per
// block before the warp tiles 100).
// Bound by instruction issue (about 60% of the slots) and the latencies
// between; the memory traffic (0.6 GB) is half of its rate.
//   * public statistics: registers -> every few chunks a warp sum into the
//     warp's FP64 shared accumulators -> one FP64 global atomic per bin per
//     CTA; whoever completes the fit's last chunk runs the public M-step into
//     the other half of a double buffer.
// No CTA waits on another CTA, nor a group on another group: every hand-off is
// "last to arrive finishes".  The mbarrier waits are bounded; on expiry the
// kernel records ST_TIMEOUT in the fit's status word and stops.
//
// A tile whose window is above the window capacity is processed "direct":
// sessions and parameters read from global memory, statistics added with FP64
// global atomics.
//
// E-step forms.  The reference evaluates PBM/UBM in closed form
// (pbm.cu:191-253, ubm.cu:185-247) and DBN/CCM through a 10x10 table of tail
// click probabilities and 80 log-space factors per session (dbn.cu:207-467,
// ccm.cu:185-478, factor.cu:73-274).  Here the same quantities are computed
// without logarithms:
//   * a rank r before the last click l has a zero z=0 factor, so its gamma/tau
//     update is a ratio independent of the tail: exactly (1, 1) for DBN and for
//     an unclicked CCM rank, (u, u) / (1-u, 1-u) with u = (1-a)t2 / ((1-a)t2 + a t3)
//     for a clicked CCM rank;
//   * for r >= l every tail that starts after r is all-unclicked and, as in the
//     reference, reads the documents at ranks 0, 1, ...; its click-probability
//     product is the r-th prefix of one forward recursion P' = P - a E,
//     E' = E g (1 - a) (E = P * examination), computed once per session;
//   * the conditional examination at ranks >= l comes from the same unnormalised
//     recursion started at the last click (nothing before it feeds it), with a
//     power-of-two rescale when P gets small (per-rank scaling), so no division
//     is needed until the final ratio.
#include <cstdint>
#include <cuda_runtime.h>
#include <cub/block/block_radix_sort.cuh>

#include "common.cuh"
#include "count_step.cuh"
#include "kernels.h"

namespace mcd {

#define FULL_MASK 0xffffffffu

// ---------------------------------------------------------------------------
// mbarrier and asynchronous-copy primitives (PTX ISA: mbarrier, cp.async)
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// try_wait that may suspend the thread until the phase completes or about
// `ns` nanoseconds pass (the suspend-time hint), instead of polling.
__device__ __forceinline__ bool mbar_try_wait_for(uint64_t* bar, uint32_t parity, uint32_t ns) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity), "r"(ns)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// Limit of one mbarrier wait, and a tile index (-1: none) for which one thread
// leaves out its arrive, so that the wait for that tile runs out with every
// copy landed: both set by set_wait_hooks for the tests of the timeout path.
__device__ unsigned long long g_wait_limit_ns = 4000000000ull;
__device__ int g_stall_tile = -1;

// Bounded wait: gives up after g_wait_limit_ns of wall-clock time (4 s unless
// a test shortened it; should the timer not advance, after 2^24 rounds of at
// least 256 ns each).
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int* status) {
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = global_ns();
    const uint64_t limit = g_wait_limit_ns;
    for (uint32_t i = 0; i < (1u << 24); i++) {
        if (mbar_try_wait_for(bar, parity, 200000u)) return true;
        if (global_ns() - t0 > limit) break;
        __nanosleep(256);
    }
    atomicOr(status, ST_TIMEOUT);
    return false;
}
// 16-byte asynchronous copies by the threads themselves (cp.async); an arrive
// that an mbarrier gets when this thread's copies so far have landed.
__device__ __forceinline__ void async_copy16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void async_arrive(uint64_t* bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void prefetch_l2(const void* src) {
    asm volatile("prefetch.global.L2 [%0];" ::"l"(src));
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL_MASK, v, o);
    return v;
}

__device__ __forceinline__ double ld_cg(const double* p) { return __ldcg(p); }

// 1 / x for normal x, one instruction (within 1 ulp).  __fdividef also scales
// operands below 2^-126, which the denominators here never are (differences
// of values clamped at 1 - 1e-6, rescaled), for three more instructions each.
__device__ __forceinline__ float rcp(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Low and high half of a packed word as exact floats plus a constant c, by
// exponent arithmetic (x < 65536 in the mantissa of 2^23): the integer to
// float conversion unit has a quarter of the rate.
__device__ __forceinline__ float lo16(uint32_t x, float c) { return __int_as_float(0x4B000000 | (x & 0xFFFFu)) - (8388608.0f - c); }
__device__ __forceinline__ float hi16(uint32_t x, float c) { return __int_as_float(0x4B000000 | (x >> 16)) - (8388608.0f - c); }

// ---------------------------------------------------------------------------
// Tiles in shared memory
// ---------------------------------------------------------------------------
// A group's shared memory holds one array of `cap` entries per kind of value:
// float atr, float sat (when satisfaction is a private statistic), uint32
// cnt16, then one bin array per private statistic.  A window starts at its
// first qd rounded down to a multiple of four (the copies are of 16 bytes,
// and the M-step takes aligned groups of four): window entry i is entry
// i + woff.  The bins are zero between tiles.
struct Layout {
    uint32_t sat_off, cnt_off, bins_off, bins2_off, bytes;  // of the arrays
};

__host__ __device__ constexpr int layout_stats(int model) { return (model == DBN || model < 0) ? 2 : 1; }

__host__ __device__ constexpr Layout make_layout(int model, int cap) {
    Layout L{};
    const uint32_t ns = (uint32_t)layout_stats(model), w4 = (uint32_t)cap * 4u;
    L.sat_off = w4;
    L.cnt_off = ns * w4;
    L.bins_off = (ns + 1u) * w4;
    L.bins2_off = L.bins_off + w4;
    L.bytes = (2u * ns + 1u) * w4;
    return L;
}

// A session as its thread holds it: five words of packed window positions
// (rank 2j in the low half of word j, 2j + 1 in the high half), each the byte
// offset 4 (i + woff) of window entry i, and the click mask.
struct Session {
    uint32_t w[MC_R / 2];
    unsigned m;
    __device__ __forceinline__ uint32_t at(int r) const { return (r & 1) ? w[r >> 1] >> 16 : w[r >> 1] & 0xFFFFu; }
    // at(l) for a lane's own l: selects, since registers cannot be indexed.
    __device__ __forceinline__ uint32_t at_lane(int l) const {
        uint32_t x = w[0];
#pragma unroll
        for (int j = 1; j < MC_R / 2; j++) x = l >= 2 * j ? w[j] : x;
        return (l & 1) ? x >> 16 : x & 0xFFFFu;
    }
};

// Statistic sinks.  A tile's bins hold 32-bit unsigned fixed point, v * 2^shift
// added with integer atomics, when the shift of its block (fx_scale) allows at
// least FX_MIN_SHIFT fraction bits; otherwise FP32 added with float atomics.
// Shared-memory float atomics are several times the cost of integer ones
// here, and at about nine adds per session they were a third of the launch.
// The fixed-point sum of a bin is exact (integer addition, any order, and any
// cut of a block into tiles); each added value carries one rounding of at most
// 2^-(shift+1).
//
// Attractiveness values are proportional to the pair's own attractiveness a,
// which ranges over several decades, so each of their adds is scaled by a
// further 2^b, b = 126 - e(a) with e(a) the biased exponent of a: a 2^b lies in
// [1/2, 1).  Every add of one pair in one tile sees the same a (the values of
// the iteration before), so the bin is one fixed-point sum with step
// 2^-(shift + b), which the M-step takes out again from the same old value.
// Pairs with a below 2^-60 (a set to 0, say) add nothing that an FP32 sum
// above 1 could hold: the M-step takes their bins as 0.
constexpr int kLeastExponent = 66;  // of an a above that

// 2^-(shift + b) from x = 2^-shift and a, 0 for a below 2^-60.
__device__ __forceinline__ float unboost(float x, float a) {
    const int e = __float_as_int(a) & 0x7F800000;
    return e >= kLeastExponent << 23 ? __int_as_float(__float_as_int(x) + e - (126 << 23)) : 0.0f;
}

// FX: fixed-point bins.  scaled(a): a 2^(shift + b) (FX), the factor of a pair's
// attractiveness terms, else a.  CAP: entries per array where
// they are fixed (a warp's memory): the arrays' offsets are then part of the
// instructions.
template <bool FX, int MODEL, int CAP>
struct StagedView {
    unsigned char* slot;  // the group's memory
    int cap;
    float scale;  // 2^shift (FX), 1 otherwise
    __device__ __forceinline__ Layout layout() const { return make_layout(MODEL, CAP ? CAP : cap); }
    __device__ __forceinline__ float a(uint32_t o) const { return *reinterpret_cast<const float*>(slot + o); }
    __device__ __forceinline__ float s(uint32_t o) const { return *reinterpret_cast<const float*>(slot + o + layout().sat_off); }
    __device__ __forceinline__ float scaled(float a) const {
        return FX ? __int_as_float((__float_as_int(a) & 0x007FFFFF) | (__float_as_int(scale) - (1 << 23))) : a;
    }
    __device__ __forceinline__ void put(unsigned char* p, float x) const {
        if (FX) atomicAdd(reinterpret_cast<unsigned*>(p), __float2uint_rn(x));
        else atomicAdd(reinterpret_cast<float*>(p), x);
    }
    __device__ __forceinline__ void add_a(uint32_t o, float x) const { put(slot + o + layout().bins_off, x); }
    __device__ __forceinline__ void add_s(uint32_t o, float x) const { put(slot + o + layout().bins2_off, x); }
};

// Direct tile: values and FP64 bins in global memory, offsets are window
// entries (scale 1).
struct DirectView {
    const float *atr, *sat;
    double* bins;
    int ns;
    static constexpr float scale = 1.0f;
    __device__ __forceinline__ float a(uint32_t o) const { return atr[o]; }
    __device__ __forceinline__ float s(uint32_t o) const { return sat[o]; }
    __device__ __forceinline__ float scaled(float a) const { return a; }
    __device__ __forceinline__ void add_a(uint32_t o, float x) const { atomicAdd(bins + (int64_t)o * ns, (double)x); }
    __device__ __forceinline__ void add_s(uint32_t o, float x) const { atomicAdd(bins + (int64_t)o * ns + 1, (double)x); }
};

// A session of a direct tile: ten window entries.
struct WideSession {
    int rl[MC_R];
    unsigned m;
    __device__ __forceinline__ uint32_t at(int r) const { return (uint32_t)rl[r]; }
    __device__ __forceinline__ uint32_t at_lane(int l) const {
        int x = rl[0];
#pragma unroll
        for (int j = 1; j < MC_R; j++) x = l >= j ? rl[j] : x;
        return (uint32_t)x;
    }
};

// Fixed point needs sum <= 2^31 for every bin: a bin takes at most one value
// per packed (session, rank) showing its pair, so at most max_occ values (the
// block's largest packed occurrence count), each below 2^ev
// (fx_value_exponent).  shift = 31 - ceil(log2 max_occ) - ev.  An
// attractiveness value is v 2^b = (v / a)(a 2^b) < v / a for a < 1, and
// fx_value_exponent bounds v / a as well as v.
constexpr int FX_MIN_SHIFT = 20;

__device__ __forceinline__ float fx_scale(int max_occ, int ev) {
    if (max_occ <= 0) return 0.0f;
    const int need = (max_occ > 1 ? 32 - __clz(max_occ - 1) : 0) + ev;
    const int shift = 31 - need;
    return shift >= FX_MIN_SHIFT ? __int_as_float((127 + shift) << 23) : 0.0f;
}

// ev with every private statistic value below 2^ev, with a factor 2 of margin
// for rounding.  DBN attractiveness a(1 - eps)/(1 - eps car) and satisfaction
// s/(1 - (1 - s) g car), the CCM unclicked attractiveness term and the PBM /
// UBM terms (a - ae)/(1 - ae) are at most 1 (car <= 1, eps <= 1, e <= 1), and
// so are their attractiveness terms divided by a.  The CCM term of a clicked
// last rank, a / (1 - (t2 (1 - a) + t3 a) car), and that term divided by a,
// are at most 1 / (1 - max(t2, t3)).
__device__ __forceinline__ int fx_value_exponent(int model, const float* pub) {
    if (model != CCM) return 1;
    const float tm = fmaxf(pub[1], pub[2]);
    const float vb = 2.0f * fmaxf(1.0f, __frcp_ru(1.0f - tm));
    const unsigned c = (unsigned)fminf(ceilf(vb), 2147483648.0f);
    return 32 - __clz(c - 1);
}

// ---------------------------------------------------------------------------
// PBM (pbm.cu:191-253): unclicked rank -> atr += (a - ae)/(1 - ae),
// exm[r] += (e - ae)/(1 - ae); clicked contributions are constant counts.
// ---------------------------------------------------------------------------
template <class Ses, class View>
__device__ __forceinline__ void estep_pbm(const Ses& ses, const View& v, const float* pub, float* acc) {
#pragma unroll
    for (int r = 0; r < MC_R; r++) {
        if (!((ses.m >> r) & 1u)) {
            const uint32_t o = ses.at(r);
            const float a = v.a(o), e = pub[r];
            const float ae = a * e, as = v.scaled(a);
            const float inv = rcp(1.0f - ae);
            v.add_a(o, (as - as * e) * inv);
            acc[r] += (e - ae) * inv;
        }
    }
}

// ---------------------------------------------------------------------------
// UBM (ubm.cu:185-247): examination slot r(r+1)/2 + prev_r (prev = 9 when no
// earlier click).  A slot written by two ranks of one session keeps the later
// rank's value; the counts of written / clicked-written slots are constants.
// ---------------------------------------------------------------------------
template <class Ses, class View>
__device__ __forceinline__ void estep_ubm(const Ses& ses, const View& v, bool valid, const float* pub, int (&key)[MC_R],
                                          float (&var)[MC_R]) {
#pragma unroll
    for (int r = 0; r < MC_R; r++) { key[r] = -1; var[r] = 0.0f; }
    if (!valid) return;
    int slot[MC_R];
    int last = 9;
#pragma unroll
    for (int r = 0; r < MC_R; r++) {
        slot[r] = r * (r + 1) / 2 + last;
        if ((ses.m >> r) & 1u) last = r;
    }
#pragma unroll
    for (int r = 0; r < MC_R; r++) {
        bool alive = true;
#pragma unroll
        for (int r2 = r + 1; r2 < MC_R; r2++) alive = alive && (slot[r2] != slot[r]);
        if (!((ses.m >> r) & 1u)) {
            const uint32_t o = ses.at(r);
            const float a = v.a(o), e = pub[slot[r]];
            const float ae = a * e, as = v.scaled(a);
            const float inv = rcp(1.0f - ae);
            v.add_a(o, (as - as * e) * inv);
            if (alive) { key[r] = slot[r]; var[r] = (e - ae) * inv; }
        }
    }
}

// Warp-level reduction of the UBM public statistics into the warp's FP64
// accumulators: for each rank, each of its r + 1 possible slots is summed over
// the lanes that chose it.
__device__ __forceinline__ void reduce_ubm_public(const int (&key)[MC_R], const float (&var)[MC_R], double* wacc) {
    int lane = threadIdx.x & 31;
    // Sessions of a tile are sorted by click mask and the slots depend only on
    // the mask, so most warps hold one key per rank in every lane: one sum
    // per rank.
    // Every lane executes every shuffle (no short-circuit around it).
    bool same = true;
#pragma unroll
    for (int r = 0; r < MC_R; r++) {
        const int k0 = __shfl_sync(FULL_MASK, key[r], 0);
        same &= key[r] == k0;
    }
    if (__all_sync(FULL_MASK, same)) {
#pragma unroll
        for (int r = 0; r < MC_R; r++) {
            if (key[r] >= 0) {  // uniform over the warp
                float v = warp_sum(var[r]);
                if (lane == 0) wacc[key[r]] += (double)v;
            }
        }
        return;
    }
#pragma unroll
    for (int r = 0; r < MC_R; r++) {
#pragma unroll
        for (int p = 0; p <= r; p++) {
            int cand = r * (r + 1) / 2 + (p == r ? 9 : p);
            unsigned hit = __ballot_sync(FULL_MASK, key[r] == cand);
            if (hit) {
                float v = warp_sum(key[r] == cand ? var[r] : 0.0f);
                if (lane == 0) wacc[cand] += (double)v;
            }
        }
    }
}

// What the DBN and CCM E-steps share.  With g the continuation after an
// unclicked document (gamma, tau_1) and gna_r = g (1 - a_r), for the last
// click's rank l:
//   car_r = a_r + gna_r car_{r+1}, car_10 = 0 (compute_exm_car), wanted at the
//     ranks after l and at l + 1;
//   Pu_j, the product of the all-unclicked tail over documents 0 .. j - 1:
//     Pu_0 = 1, Pu' = Pu - a Eu, Eu_0 = 1, Eu' = Eu gna.  A rank r >= l has the
//     tail R_r = Pu_{9-r}.
// Both run in one loop: two chains in flight.
//
// At a rank after l, with (P, E) the conditional examination (from the last
// click on) and eps the unconditional one: h = E / (P - g E (1 - R)) gives the
// public terms g R h (numerator) and (1 - g) h + g R h (denominator), summed as h
// and R h: as h and (1 - R) h, a small R would be lost to cancellation where
// documents are all attractive (a = 0.999: 2e-4 of the value).  The pair's term is
// a (1 - eps)/(1 - eps car).
//
// The ranks run straight through for all lanes, without a branch on a lane's
// own l: E is 0 up to its last click, so that h is 0 and P stays 1, takes the
// value E_l at rank l + 1, and only the add is predicated.  (Sessions are
// sorted by l, but a tile of rare queries has one chunk with every l in it, and
// branches on l kept the ranks' chains from overlapping.)  Three ranks at a
// time are skipped when no lane has a last click before them.
struct Ranks {
    float a[MC_R], gna[MC_R], car[MC_R], Pu[MC_R];
    float P, E, eps, car_l, R_l;
};

template <class Ses, class View>
__device__ __forceinline__ void load_ranks(Ranks& k, const Ses& ses, const View& v, float g) {
#pragma unroll
    for (int r = 0; r < MC_R; r++) {
        k.a[r] = v.a(ses.at(r));
        k.gna[r] = g * (1.0f - k.a[r]);
    }
    float c = 0.0f, pu = 1.0f, eu = 1.0f;
#pragma unroll
    for (int j = 0; j < MC_R; j++) {
        const int r = MC_R - 1 - j;
        k.Pu[j] = pu;
        if (r > 0) {
            c = fmaf(k.gna[r], c, k.a[r]);
            k.car[r] = c;
            pu = fmaf(-k.a[j], eu, pu);
            eu *= k.gna[j];
        }
    }
    k.P = k.eps = k.R_l = 1.0f;
    k.E = k.car_l = 0.0f;
}

// Rank r >= 1 of a lane with last click l (10: none) and E_l.
template <class Ses, class View>
__device__ __forceinline__ void rank_after(Ranks& k, const Ses& ses, const View& v, int r, int l, float g, float E_l, float& sh,
                                           float& srh) {
    const float R = k.Pu[MC_R - 1 - r];
    if (l == r - 1) {
        k.E = E_l;
        k.car_l = k.car[r];
        k.R_l = k.Pu[MC_R - r];
    }
    const float h = k.E * rcp(fmaf(k.E, fmaf(g, R, -g), k.P));
    sh += h;
    srh = fmaf(h, R, srh);
    const float x = v.scaled(k.a[r]) * (1.0f - k.eps) * rcp(1.0f - k.eps * k.car[r]);
    if (l < r) v.add_a(ses.at(r), x);
    k.P = fmaf(-k.a[r], k.E, k.P);
    k.E *= k.gna[r];
    // Per-rank scaling: a rank multiplies P by at least 1 - (1 - 1e-6)^2 =
    // 2e-6, and P - g E (1 - R) is at least that share of P, so a look at
    // every third rank keeps both normal.
    if (r % 3 == 0 && r < MC_R - 1 && k.P < 1e-4f) {
        k.P *= 1.8446744e19f;
        k.E *= 1.8446744e19f;
    }
}

// Last click of a lane (10: none, a lane without a session) and the smallest
// one of the warp.
__device__ __forceinline__ int last_click(unsigned m, int& l_min) {
    const int l = m ? 31 - __clz(m) : MC_R;
    l_min = __reduce_min_sync(FULL_MASK, l);
    return l;
}

// ---------------------------------------------------------------------------
// DBN (dbn.cu:207-467); acc: sum of h and of R h.  Ranks before the last click
// contribute exactly (1, 1) each and a session without clicks (10, 10) and
// nothing else: constants of the fit, added at upload (model.cu).
// ---------------------------------------------------------------------------
template <class Ses, class View>
__device__ __forceinline__ void estep_dbn(const Ses& ses, const View& v, float g, float* acc) {
    int l_min;
    const int l = last_click(ses.m, l_min);
    Ranks k;
    load_ranks(k, ses, v, g);
    const uint32_t ol = ses.at_lane(l);
    const float sl = v.s(ol), cs = 1.0f - sl, E_l = cs * g;
#pragma unroll
    for (int q = 0; q < 3; q++) {
        if (l_min <= 3 * q + 2) {
#pragma unroll
            for (int r = 3 * q + 1; r <= 3 * q + 3; r++) {
                k.eps *= g * (1.0f - k.a[r - 1] * v.s(ses.at(r - 1)));  // g (1 - a) + g a (1 - s)
                rank_after(k, ses, v, r, l, g, E_l, acc[0], acc[1]);
            }
        } else {
#pragma unroll
            for (int r = 3 * q + 1; r <= 3 * q + 3; r++) k.eps *= g * (1.0f - k.a[r - 1] * v.s(ses.at(r - 1)));
        }
    }
    // The last click: satisfaction, and gamma with h = (1 - s) / (1 - g (1 - s)(1 - R)).
    if (l < MC_R) {
        const float h = cs * rcp(fmaf(cs, fmaf(g, k.R_l, -g), 1.0f));
        acc[0] += h;
        acc[1] = fmaf(h, k.R_l, acc[1]);
        v.add_s(ol, v.scale * (sl * rcp(1.0f - E_l * k.car_l)));
    }
}

// ---------------------------------------------------------------------------
// CCM (ccm.cu:185-478); acc: sum of h and of R h (tau_1), then the tau_2 and
// tau_3 numerators and denominators.
// ---------------------------------------------------------------------------
template <class Ses, class View>
__device__ __forceinline__ void estep_ccm(const Ses& ses, const View& v, float t1, float t2, float t3, float* acc) {
    int l_min;
    const int l = last_click(ses.m, l_min);
    Ranks k;
    load_ranks(k, ses, v, t1);
    // Clicks before the last one: only the tau_2 / tau_3 split depends on the
    // parameters: u = x / (x + y) and 1 - u = y / (x + y), each from its own
    // numerator (1 - u formed by subtraction loses the small tau_3 share to
    // cancellation when tau_3 is near 0).
    for (unsigned rest = ses.m & ~(1u << l); rest; rest &= rest - 1u) {
        const float a = v.a(ses.at_lane(31 - __clz(rest & -rest)));
        const float x = (1.0f - a) * t2, y = a * t3;
        const float inv = rcp(x + y);
        const float p = x * inv, q = y * inv;
        acc[2] += p; acc[3] += p;
        acc[4] += q; acc[5] += q;
    }
    const uint32_t ol = ses.at_lane(l);
    const float al = v.a(ol), ial = 1.0f - al, E_l = __fadd_rn(__fmul_rn(t2, ial), __fmul_rn(t3, al));
    // (1 - a) t1 + a ((1 - a) t2 + a t3), rounded as it always has been: values
    // are compared with those of earlier fits.
    auto step = [&](int r) {
        const float a = k.a[r], ia = 1.0f - a;
        const float in = fmaf(ia, t2, __fmul_rn(a, t3));
        k.eps *= r < 2 ? fmaf(a, in, k.gna[r]) : fmaf(ia, t1, __fmul_rn(a, in));
    };
#pragma unroll
    for (int q = 0; q < 3; q++) {
        if (l_min <= 3 * q + 2) {
#pragma unroll
            for (int r = 3 * q + 1; r <= 3 * q + 3; r++) {
                step(r - 1);
                rank_after(k, ses, v, r, l, t1, E_l, acc[0], acc[1]);
            }
        } else {
#pragma unroll
            for (int r = 3 * q + 1; r <= 3 * q + 3; r++) step(r - 1);
        }
    }
    if (l == MC_R) return;
    const float R = k.R_l;
    const float k2 = 1.0f - t2 * (1.0f - R), k3 = 1.0f - t3 * (1.0f - R);
    const float B = rcp(ial * k2 + al * k3);
    acc[2] += ial * t2 * R * B;
    acc[3] += ial * k2 * B;
    acc[4] += al * t3 * R * B;
    acc[5] += al * k3 * B;
    v.add_a(ol, v.scaled(al) * rcp(1.0f - E_l * k.car_l));
}

// Registers a warp's lanes sum the public statistics in (UBM: none, its
// statistics go to the warp's accumulators chunk by chunk) and the bins of the
// fit that they end in: DBN and CCM statistic q to pub_bins[q], PBM and UBM
// numerator k to pub_bins[2 k].
__host__ __device__ constexpr int acc_regs(int model) { return model == DBN ? 2 : model == CCM ? 6 : model == UBM ? 0 : MC_R; }
__device__ __forceinline__ int acc_count(int model) { return model == UBM ? MC_UBM_SLOTS : acc_regs(model); }

// Sums of h and R h as numerator and denominator terms: g R h and (1 - g) h + g R h.
// v: statistic q of lane q.
__device__ __forceinline__ double finish_acc(int model, int q, double v, float g) {
    if (model != DBN && model != CCM) return v;
    const double h = __shfl_sync(FULL_MASK, v, 0), rh = (double)g * __shfl_sync(FULL_MASK, v, 1);
    return q == 0 ? rh : q == 1 ? fma(1.0 - (double)g, h, rh) : v;
}

// ---------------------------------------------------------------------------
// M-step of one qd from its counts and variable statistics.
//   PBM / UBM / DBN attractiveness: (1 + clicks + v0) / (2 + occurrences)
//   CCM attractiveness:             (1 + clicks + v0) / (2 + occurrences + clicks)
//   DBN satisfaction, parity:       (1 + unclicked + v1) / (2 + clicks + 2 unclicked)
//   DBN satisfaction, clean:        (1 + v1) / (2 + clicks)
// ---------------------------------------------------------------------------
// One qd of a query within one block in FP32 (the quotient is a product with
// the 1-ulp reciprocal): c the packed counts (occurrences, clicks << 16), v0
// and v1 the statistics.
__device__ __forceinline__ float mstep_atr(bool ccm, uint32_t c, float v0) {
    const float num = hi16(c, 1.0f) + v0, den = lo16(c, 2.0f);
    return fminf(num * rcp(ccm ? den + hi16(c, 0.0f) : den), MC_TOP);
}

__device__ __forceinline__ float mstep_sat(int mode, uint32_t c, float v1) {
    const float clk = hi16(c, 0.0f), un = mode == PARITY ? lo16(c, 0.0f) - clk : 0.0f;
    return fminf((1.0f + un + v1) * rcp(fmaf(2.0f, un, 2.0f + clk)), MC_TOP);
}

__device__ __forceinline__ void mstep_qd_d(int model, int mode, uint2 cnt, double v0, double v1, float* atr, float* sat) {
    double occ = (double)cnt.x, clk = (double)cnt.y;
    double den = model == CCM ? 2.0 + occ + clk : 2.0 + occ;
    double v = (1.0 + clk + v0) / den;
    *atr = (float)(v < (double)MC_TOP ? v : (double)MC_TOP);
    if (model == DBN) {
        double un = occ - clk;
        double sn = mode == PARITY ? 1.0 + un + v1 : 1.0 + v1;
        double sd = mode == PARITY ? 2.0 + clk + 2.0 * un : 2.0 + clk;
        double w = sn / sd;
        *sat = (float)(w < (double)MC_TOP ? w : (double)MC_TOP);
    }
}

// Public M-step of a fit whose last chunk has finished (one warp).  Everything
// it reads is loaded at once: the launch waits for this chain.
__device__ void finalize_public(const FitDev& f, int lane) {
    const int it = *(volatile int*)f.iter;
    double num[2], den[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int k = lane + 32 * h;
        if (k < f.n_pub) {
            num[h] = f.pub_const[2 * k] + ld_cg(f.pub_bins + 2 * k);
            den[h] = f.pub_const[2 * k + 1] + ld_cg(f.pub_bins + 2 * k + 1);
        }
    }
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int k = lane + 32 * h;
        if (k < f.n_pub) {
            const double v = num[h] / den[h];
            f.pub_theta[((it + 1) & 1) * MC_MAX_PUB + k] = (float)(v < (double)MC_TOP ? v : (double)MC_TOP);
            f.pub_bins[2 * k] = 0.0;
            f.pub_bins[2 * k + 1] = 0.0;
        }
    }
    if (lane == 0) {
        *f.tiles_done = 0;
        *(volatile int*)f.iter = it + 1;  // read by later launches only
    }
    __syncwarp();
}

// Adds a warp's sums (statistic q in v of lane q, q + 32 in v2) to the fit's
// public bins, counts its chunks, and runs the public M-step if they were the
// fit's last.  All lanes.
__device__ void flush_public(const FitDev& f, int model, int lane, double v, double v2, float g, unsigned chunks) {
    const int n = acc_count(model), step = (model == DBN || model == CCM) ? 1 : 2;
    v = finish_acc(model, lane, v, g);
    if (lane < n && v != 0.0) atomicAdd(f.pub_bins + step * lane, v);
    if (lane + 32 < n && v2 != 0.0) atomicAdd(f.pub_bins + step * (lane + 32), v2);
    __threadfence();
    __syncwarp();
    unsigned last = 0;
    if (lane == 0) last = atomicAdd(f.tiles_done, chunks) + chunks == (unsigned)f.n_chunks;
    last = __shfl_sync(FULL_MASK, last, 0);
    if (last) {
        __threadfence();
        finalize_public(f, lane);
    }
}

template <int MODEL>
__device__ __forceinline__ int model_of(const FitDev& f) { return MODEL >= 0 ? MODEL : f.model; }

// E-step chunks of a tile (at least one, so that every tile counts).
__device__ __forceinline__ int tile_chunks(int sessions) { return sessions > 32 ? (sessions + 31) >> 5 : 1; }

// One chunk of sessions into the view's bins and the accumulators.
template <int MODEL, class Ses, class View>
__device__ __forceinline__ void estep_chunk(int model, const Ses& ses, const View& v, bool valid, const float* pub, float* acc,
                                            double* wacc) {
    if (model == DBN) {
        if (MODEL == DBN || MODEL < 0) estep_dbn(ses, v, pub[0], acc);
    } else if (model == CCM) {
        if (MODEL == CCM || MODEL < 0) estep_ccm(ses, v, pub[0], pub[1], pub[2], acc);
    } else if (model == PBM) {
        if ((MODEL == PBM || MODEL < 0) && valid) estep_pbm(ses, v, pub, acc);
    } else if (MODEL == UBM || MODEL < 0) {
        int key[MC_R];
        float var[MC_R];
        estep_ubm(ses, v, valid, pub, key, var);
        reduce_ubm_public(key, var, wacc);
    }
}

// Entries of a warp's memory (a narrow tile's arrays).
__host__ __device__ constexpr int narrow_cap(int model) { return layout_stats(model) > 1 ? 408 : 680; }

// A chunk of a tile that needs FP32 bins, and a chunk of a direct tile: rarer, out
// of line so that the hot loop stays small in the instruction cache.
template <int MODEL>
__device__ __noinline__ void estep_chunk_other(int model, const Session ses, unsigned char* slot, int cap, bool valid,
                                               const float* pub, float* acc, double* wacc) {
    const StagedView<false, MODEL, 0> v{slot, cap, 1.0f};
    estep_chunk<MODEL>(model, ses, v, valid, pub, acc, wacc);
}

template <int MODEL>
__device__ __noinline__ void estep_chunk_direct(int model, const FitDev& f, const TileDev& tile, double* bins, int sl,
                                                const float* pub, float* acc, double* wacc) {
    WideSession ses;
    ses.m = 0;
    bool ok = sl < tile.s_count;
#pragma unroll
    for (int r = 0; r < MC_R; r++) {
        ses.rl[r] = 0;
        if (sl < tile.s_count) {
            const int64_t p = (int64_t)__ldg(f.pidx + (int64_t)r * f.stride + tile.s_begin + sl) - tile.qd_begin;
            if (p < 0 || p >= tile.qd_count) {
                atomicOr(f.status, ST_BAD_INDEX);
                ok = false;
            } else {
                ses.rl[r] = (int)p;
            }
        }
    }
    if (ok) ses.m = __ldg(f.click + tile.s_begin + sl);
    const DirectView v{f.atr + tile.qd_begin, f.sat ? f.sat + tile.qd_begin : nullptr, bins, private_stats(model)};
    estep_chunk<MODEL>(model, ses, v, ok, pub, acc, wacc);
}

// Chunks whose public statistics a lane sums in FP32 before they are folded
// into the warp's FP64 accumulators.
constexpr int kFoldChunks = 8;
constexpr int kWarps = FUSED_THREADS / 32;

// Doubles a warp keeps its public sums in, floats a group keeps the public
// values in.
__host__ __device__ constexpr int pub_slots(int model) { return model == DBN ? 2 : model == CCM ? 6 : model == PBM ? MC_R : 56; }

// A folded split tile that has not been counted: the query, its counter, the fit.
struct OpenSplit {
    SplitDev split;
    unsigned* count;
    int fit;
};

// The CTA's state in shared memory, beside the tiles' memory.  What the loop
// over tiles needs now and then stays here: at 80 registers the E-step has none
// to spare, and a spill in it costs more (16M DBN sessions: up to 0.04 ms per
// iteration with the same state in registers).
template <int MODEL>
struct Shared {
    double wacc[kWarps][pub_slots(MODEL)];              // each warp's public sums, statistic q
    alignas(16) SplitDev split[kWarps];                 // per group, as the arrays below: of a split tile
    alignas(16) TileDev tile[kWarps][3];                // the k-th tile in [k % 3]
    FitDev fit[kWarps];
    uint64_t full[kWarps + 1];                          // mbarriers: per warp, and the CTA's
    float pub[kWarps][pub_slots(MODEL)];                // public values, fixed for the launch
    int index[kWarps][3];                               // of the tiles
    OpenSplit open[kWarps];                             // each warp's last fold, not counted yet
    int warp_fit[kWarps], abort;
    int last;                                           // a wide split tile was its query's last
    unsigned warp_chunks[kWarps];
};

template <int MODEL>
__device__ __forceinline__ Shared<MODEL>& cta_shared() {
    __shared__ Shared<MODEL> sh;
    return sh;
}

// M-step of a split query's pairs first, first + step, ..., whose tiles have all
// been folded; clears its bins.
template <int MODEL>
__device__ __forceinline__ void mstep_split(const FitDev& f, const SplitDev& sp, int first, int step) {
    const int model = model_of<MODEL>(f), ns = private_stats(model);
    double* const gb = f.split_bins + sp.bin_offset;
    for (int i = first; i < sp.qd_count; i += step) {
        int64_t q = sp.qd_begin + i;
        uint2 cn = __ldg(f.cnt + q);
        double v0 = ld_cg(gb + (int64_t)i * ns);
        double v1 = ns > 1 ? ld_cg(gb + (int64_t)i * ns + 1) : 0.0;
        if (sp.in_block) {  // exact sums of one scale: as an owned tile's bins
            const uint32_t c = __ldg(f.cnt16 + q);
            f.atr[q] = mstep_atr(model == CCM, c, (float)v0);
            if (ns > 1) f.sat[q] = mstep_sat(f.mode, c, (float)v1);
        } else {
            mstep_qd_d(model, f.mode, cn, v0, v1, f.atr + q, ns > 1 ? f.sat + q : nullptr);
        }
        gb[(int64_t)i * ns] = 0.0;
        if (ns > 1) gb[(int64_t)i * ns + 1] = 0.0;
    }
}

// A narrow split tile's fold counts once its FP64 adds are done; the warp does
// that after its next chunk (or before its next fold, or at the end), when the
// fence no longer waits for them.  The warp that counts the query's last tile
// runs the query's M-step.
template <int MODEL>
__device__ __noinline__ void count_split(const FitDev* __restrict__ fits) {
    const int lane = threadIdx.x & 31;
    const OpenSplit& o = cta_shared<MODEL>().open[threadIdx.x >> 5];
    __threadfence();
    __syncwarp();
    unsigned last = 0;
    if (lane == 0) last = atomicAdd(o.count, 1u) + 1 == (unsigned)o.split.n_tiles;
    last = __shfl_sync(FULL_MASK, last, 0);
    if (!last) return;
    __threadfence();
    mstep_split<MODEL>(fits[o.fit], o.split, lane, 32);
    if (lane == 0) *o.count = 0;
    __syncwarp();
}

// A CTA counts its fold of a wide split tile (split[0]), and the one that counts
// the query's last runs its M-step.
template <int MODEL>
__device__ __noinline__ void count_wide_split(const FitDev& f) {
    Shared<MODEL>& sh = cta_shared<MODEL>();
    const SplitDev& sp = sh.split[0];
    unsigned* const count = f.split_count + sp.local;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) sh.last = atomicAdd(count, 1u) + 1 == (unsigned)sp.n_tiles;
    __syncthreads();
    if (!sh.last) return;
    __threadfence();
    mstep_split<MODEL>(f, sp, threadIdx.x, blockDim.x);
    if (threadIdx.x == 0) *count = 0;
}

// Adds the sums of a warp (and clears them) to its fit's public bins.
template <int MODEL>
__device__ __noinline__ void flush_warp(const FitDev& f, unsigned chunks, float g) {
    constexpr int NP = pub_slots(MODEL);
    const int lane = threadIdx.x & 31;
    double* const w = cta_shared<MODEL>().wacc[threadIdx.x >> 5];
    __syncwarp();
    const double v = lane < NP ? w[lane] : 0.0, v2 = lane + 32 < NP ? w[lane + 32] : 0.0;
    __syncwarp();
    if (lane < NP) w[lane] = 0.0;
    if (lane + 32 < NP) w[lane + 32] = 0.0;
    flush_public(f, model_of<MODEL>(f), lane, v, v2, g, chunks);
    __syncwarp();
}

// The tiles [t_begin, t_end): ONE, a group is one warp and its tiles are
// narrow; otherwise the CTA.
template <int MODEL, bool ONE>
__device__ __forceinline__ void run_tiles(const FitDev* __restrict__ fits, const TileDev* __restrict__ tiles, int t_begin, int t_end,
                                          const SplitDev* __restrict__ splits, unsigned* queue, int window_max, int cap,
                                          int* const status) {
    extern __shared__ __align__(128) unsigned char smem[];
    Shared<MODEL>& sh = cta_shared<MODEL>();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n_warps = blockDim.x >> 5;
    const int group_warps = ONE ? 1 : n_warps, groups = ONE ? n_warps : 1;
    const int group = ONE ? warp : 0, gw = ONE ? 0 : warp;  // gw: this warp in its group
    const int n_groups = groups * (int)gridDim.x;
    const int group_cap = ONE ? narrow_cap(MODEL) : cap;
    const Layout L = make_layout(MODEL, group_cap);
    unsigned char* const slot = smem + (size_t)group * L.bytes;
    uint64_t* const bar = &sh.full[ONE ? warp : kWarps];
    auto group_sync = [&]() {
        if (ONE) __syncwarp();
        else __syncthreads();
    };
    auto group_all = [&](bool ok) { return ONE ? (bool)__all_sync(FULL_MASK, ok) : (bool)__syncthreads_and(ok); };
    __syncthreads();  // the tiles before, if any, are done with the memory
    for (int i = gw * 32 + lane; i < (int)((L.bytes - L.bins_off) / 16); i += group_warps * 32)
        reinterpret_cast<uint4*>(slot + L.bins_off)[i] = make_uint4(0u, 0u, 0u, 0u);
    if (gw == 0 && lane == 0) mbar_init(bar, group_warps * 32);

    // A chunk of sessions per warp, behind the tiles' memory.
    unsigned char* const my_chunk = smem + make_layout(MODEL, cap).bytes + (size_t)warp * kChunkBytes;
    auto fetch_chunk = [&](const unsigned char* src) {
        async_copy16(my_chunk + lane * 16, src + lane * 16);
        if (lane < kChunkBytes / 16 - 32) async_copy16(my_chunk + (lane + 32) * 16, src + (lane + 32) * 16);
    };

    // Tile indices (the group's last warp) come in runs of consecutive tiles
    // (guided self-scheduling: a run is about 1/4 of the queue left per group,
    // 1 to 8 tiles, estimated from the position this group last took), so a
    // group's tiles are mostly neighbours.  The first run is the group's own by
    // its index; a later run's counter value is asked for with the last tile of
    // the run before and used one tile later.  Queues of at most two tiles per
    // group are all the groups' own (thousands of groups asking one counter at
    // once took 3 us: 2M sessions 45.9 -> 40.8 us per iteration).
    auto run_length = [&](int left) { return max(1, min(8, left / (4 * n_groups))); };
    const bool two_rounds = t_end - t_begin <= 2 * n_groups;
    const int first_run = two_rounds ? 1 : run_length(t_end - t_begin);
    // After wide tiles the last CTAs come first: those have had the fewest.
    const int cta = ONE && t_begin > 0 ? (int)(gridDim.x - 1 - blockIdx.x) : (int)blockIdx.x;
    int run_next = t_begin + (cta * groups + group) * first_run, run_end = run_next + first_run;
    unsigned asked = 0;
    // The next tile's descriptor on its way to tile[slot3].
    auto take_tile = [&](int slot3) {
        if (run_next >= run_end) {
            if (two_rounds) {
                run_next = run_end - 1 + n_groups;
                run_end = run_next + 1;
            } else {
                const int len = run_length(t_end - run_end);
                run_next = t_begin + n_groups * first_run + (int)__shfl_sync(FULL_MASK, asked, 0);
                run_end = run_next + len;
            }
        }
        const int t = run_next++;
        if (run_next == run_end && !two_rounds && lane == 0) asked = atomicAdd(queue, (unsigned)run_length(t_end - run_end));
        TileDev* const to = &sh.tile[group][slot3];
        if (t < t_end) {
            if (lane < 3) async_copy16(reinterpret_cast<unsigned char*>(to) + lane * 16, reinterpret_cast<const unsigned char*>(tiles + t) + lane * 16);
        } else if (lane == 0) {
            to->s_count = -1;  // the end of this group's tiles
        }
        if (lane == 0) sh.index[group][slot3] = t;
    };
    // The group's last warp, which has the fewest chunks, looks ahead (the first
    // one doing so: 1.6M DBN sessions in queries of 200 over 600 pairs 74 us per
    // iteration, the last 69; of 42 over 420 pairs 162 and 140).
    const bool scout = gw == group_warps - 1;
    if (scout) {
        take_tile(0);
        take_tile(1);
        async_wait_all();
    }

    // This warp's public sums of the current fit.
    constexpr int NA = acc_regs(MODEL < 0 ? PBM : MODEL) > 0 ? acc_regs(MODEL < 0 ? PBM : MODEL) : 1;
    float acc[NA];
#pragma unroll
    for (int q = 0; q < NA; q++) acc[q] = 0.0f;
    auto fold = [&]() {
        if constexpr (MODEL != UBM) {
#pragma unroll
            for (int q = 0; q < NA; q++) {
                const float v = warp_sum(acc[q]);
                if (lane == 0 && v != 0.0f) sh.wacc[warp][q] += (double)v;
                acc[q] = 0.0f;
            }
        }
    };
    int cur_fit = -1;  // the fit in fit[], pub[], and of the sums
    unsigned cur_chunks = 0;
    bool open = false;

    for (int k = 0, k3 = 0;; k++, k3 = k3 == 2 ? 0 : k3 + 1) {
        const TileDev& tile = sh.tile[group][k3];
        group_sync();  // the tile before is done: its memory is free
        if (tile.s_count < 0) break;
        const bool direct = !ONE && tile.qd_count > window_max;
        const int woff = (int)(tile.qd_begin & 3), wend = woff + tile.qd_count;
        if (tile.fit != cur_fit) {
            if (cur_chunks) {
                fold();
                flush_warp<MODEL>(sh.fit[group], cur_chunks, sh.pub[group][0]);
                cur_chunks = 0;
            }
            // For every warp of the group, also one that the former fit's tiles
            // had no chunk for: fit[] and pub[] are written anew below.
            if (cur_fit >= 0) group_sync();
            if (gw == 0) {
                const FitDev& fg = fits[tile.fit];
                if (lane < (int)(sizeof(FitDev) / 8))
                    reinterpret_cast<uint64_t*>(&sh.fit[group])[lane] = reinterpret_cast<const uint64_t*>(&fg)[lane];
                const int it = *(volatile int*)fg.iter;
                for (int q = lane; q < fg.n_pub; q += 32) sh.pub[group][q] = __ldcg(fg.pub_theta + (it & 1) * MC_MAX_PUB + q);
            }
            group_sync();
            cur_fit = tile.fit;
        }
        const FitDev& f = sh.fit[group];
        const float* const pub = sh.pub[group];
        const int model = model_of<MODEL>(f);
        const int n_sess = direct ? tile.s_count : tile.s_packed;
        const int n_chunks = tile_chunks(n_sess);
        const bool packed = !direct && n_sess > 0;
        const unsigned char* chunk = f.tblk + tile.blk_off + (int64_t)gw * kChunkBytes;
        {
            const int64_t a0 = tile.qd_begin & ~(int64_t)3;
            const int n16 = direct ? 0 : (wend + 3) >> 2;
            const float* const sat = layout_stats(MODEL) > 1 ? f.sat : nullptr;
            for (int i = gw * 32 + lane; i < n16; i += group_warps * 32) {
                unsigned char* const to = slot + i * 16;
                async_copy16(to, f.atr + a0 + i * 4);
                if (sat) async_copy16(to + L.sat_off, sat + a0 + i * 4);
                if (tile.split < 0) async_copy16(to + L.cnt_off, f.cnt16 + a0 + i * 4);
            }
            if (tile.split >= 0 && gw == 0 && lane < (int)sizeof(SplitDev) / 16)
                async_copy16(reinterpret_cast<unsigned char*>(&sh.split[group]) + lane * 16,
                             reinterpret_cast<const unsigned char*>(splits + tile.split) + lane * 16);
            if (packed && gw < n_chunks) fetch_chunk(chunk);
            // One arrive is left out for the tests of the timeout path.
            if (gw != 0 || lane != 0 || sh.index[group][k3] != g_stall_tile) async_arrive(bar);
        }
        const int next = k3 == 2 ? 0 : k3 + 1;
        if (scout) take_tile(next == 2 ? 0 : next + 1);
        const float sc = fx_scale(tile.max_occ, fx_value_exponent(model, pub));  // 2^shift of the bins, 0: FP32
        // Every lane observes the completed phase itself.
        bool ok = mbar_wait(bar, (uint32_t)k & 1u, status);
        ok = group_all(ok);  // the group leaves together
        if (!ok) {
            sh.abort = 1;
            async_wait_all();  // copies still in flight
            break;
        }
        if (scout) {  // the next tile's values and sessions to L2 (when it is of the same fit)
            const TileDev& n = sh.tile[group][next];
            if (n.s_count >= 0 && n.fit == cur_fit && n.qd_count <= window_max) {
                const unsigned char* const na = reinterpret_cast<const unsigned char*>(f.atr + n.qd_begin);
                const unsigned char* const ns = reinterpret_cast<const unsigned char*>(f.sat + n.qd_begin);
                const unsigned char* const nc = reinterpret_cast<const unsigned char*>(f.cnt16 + n.qd_begin);
                for (int i = lane * 128; i < n.qd_count * 4; i += 32 * 128) {
                    prefetch_l2(na + i);
                    if (layout_stats(MODEL) > 1 && f.sat) prefetch_l2(ns + i);
                    prefetch_l2(nc + i);
                }
                for (int i = lane * 128; i < (n.s_packed + 31) / 32 * kChunkBytes; i += 32 * 128) prefetch_l2(f.tblk + n.blk_off + i);
            }
        }

        for (int c = gw; c < n_chunks; c += group_warps, chunk += group_warps * kChunkBytes) {
            const int sl = (c << 5) + lane;
            Session ses;
            if (packed) {
                if (c != gw) {  // the first chunk came with the tile's values
                    async_wait_all();
                    __syncwarp();
                }
                const uint32_t* const words = reinterpret_cast<const uint32_t*>(my_chunk) + lane;
#pragma unroll
                for (int q = 0; q < MC_R / 2; q++) ses.w[q] = words[q * 32];
                ses.m = reinterpret_cast<const uint16_t*>(my_chunk + 5 * 128)[lane];
                __syncwarp();
                if (c + group_warps < n_chunks) fetch_chunk(chunk + group_warps * kChunkBytes);
            }
            if (packed && sc != 0.0f) {
                const StagedView<true, MODEL, ONE ? narrow_cap(MODEL) : 0> v{slot, group_cap, sc};
                estep_chunk<MODEL>(model, ses, v, sl < n_sess, pub, acc, sh.wacc[warp]);
            } else if (packed && (MODEL == CCM || MODEL < 0)) {
                // FP32 bins: CCM's as soon as tau_2 or tau_3 is near 1 (out of line,
                // as below, 1.6M sessions with two clicks each took 78 in place of
                // 55 us per iteration).
                const StagedView<false, MODEL, ONE ? narrow_cap(MODEL) : 0> v{slot, group_cap, 1.0f};
                estep_chunk<MODEL>(model, ses, v, sl < n_sess, pub, acc, sh.wacc[warp]);
            } else if (packed || direct) {
                // The other kinds get a copy of the sums: an array whose
                // address is passed on does not stay in registers.
                float t[NA];
#pragma unroll
                for (int q = 0; q < NA; q++) t[q] = acc[q];
                if (direct) {
                    estep_chunk_direct<MODEL>(model, f, tile, f.split_bins + sh.split[group].bin_offset, sl, pub, t, sh.wacc[warp]);
                } else {
                    estep_chunk_other<MODEL>(model, ses, slot, group_cap, sl < n_sess, pub, t, sh.wacc[warp]);
                }
#pragma unroll
                for (int q = 0; q < NA; q++) acc[q] = t[q];
            }
            if ((++cur_chunks & (kFoldChunks - 1)) == 0) fold();
            if (open) {
                count_split<MODEL>(fits);
                open = false;
            }
        }
        if (direct) __threadfence();  // statistics in global memory, before the split counter is raised
        group_sync();  // the bins are complete

        const int ns = private_stats(model);
        const float inv = sc != 0.0f ? rcp(sc) : 0.0f;  // 2^-shift, exact
        if (tile.split < 0) {
            for (int i = (gw * 32 + lane) * 4; i < wend; i += group_warps * 128) {
                unsigned char* const p = slot + i * 4;
                const uint4 c = *reinterpret_cast<const uint4*>(p + L.cnt_off);
                uint4 b = *reinterpret_cast<const uint4*>(p + L.bins_off);
                const float4 o = *reinterpret_cast<const float4*>(p);
                const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
                *reinterpret_cast<uint4*>(p + L.bins_off) = zero;
                const bool ccm = model == CCM;
                auto val_a = [&](uint32_t x, float a) { return sc != 0.0f ? __uint2float_rn(x) * unboost(inv, a) : __uint_as_float(x); };
                auto val = [&](uint32_t x) { return sc != 0.0f ? __uint2float_rn(x) * inv : __uint_as_float(x); };
                float4 x;
                x.x = mstep_atr(ccm, c.x, val_a(b.x, o.x));
                x.y = mstep_atr(ccm, c.y, val_a(b.y, o.y));
                x.z = mstep_atr(ccm, c.z, val_a(b.z, o.z));
                x.w = mstep_atr(ccm, c.w, val_a(b.w, o.w));
                const int64_t q = tile.qd_begin - woff + i;
                const bool whole = i >= woff && i + 4 <= wend;
                auto store = [&](float* dst) {
                    if (whole) {
                        *reinterpret_cast<float4*>(dst + q) = x;
                    } else {
                        if (i >= woff) dst[q] = x.x;
                        if (i + 1 >= woff && i + 1 < wend) dst[q + 1] = x.y;
                        if (i + 2 >= woff && i + 2 < wend) dst[q + 2] = x.z;
                        if (i + 3 >= woff && i + 3 < wend) dst[q + 3] = x.w;
                    }
                };
                store(f.atr);
                if (layout_stats(MODEL) > 1 && ns > 1) {
                    b = *reinterpret_cast<const uint4*>(p + L.bins2_off);
                    *reinterpret_cast<uint4*>(p + L.bins2_off) = zero;
                    x.x = mstep_sat(f.mode, c.x, val(b.x));
                    x.y = mstep_sat(f.mode, c.y, val(b.y));
                    x.z = mstep_sat(f.mode, c.z, val(b.z));
                    x.w = mstep_sat(f.mode, c.w, val(b.w));
                    store(f.sat);
                }
            }
        } else {
            if (ONE && open) count_split<MODEL>(fits);  // the split tile before
            double* const gb = f.split_bins + sh.split[group].bin_offset;
            if (!direct) {
                for (int i = gw * 32 + lane; i < tile.qd_count; i += group_warps * 32)
                    for (int q = 0; q < ns; q++) {
                        unsigned char* const p = slot + (i + woff) * 4;
                        unsigned* const bin = reinterpret_cast<unsigned*>(p + (q ? L.bins2_off : L.bins_off));
                        const unsigned x = *bin;
                        if (x == 0u) continue;
                        *bin = 0u;
                        const float step = q == 0 ? unboost(inv, *reinterpret_cast<const float*>(p)) : inv;
                        const double v = sc != 0.0f ? (double)x * (double)step : (double)__uint_as_float(x);
                        if (v != 0.0) atomicAdd(gb + (int64_t)i * ns + q, v);
                    }
            }
            if (ONE) {
                if (lane == 0) sh.open[warp] = OpenSplit{sh.split[group], f.split_count + sh.split[group].local, tile.fit};
                open = true;
            } else {
                count_wide_split<MODEL>(f);
            }
        }
    }
    if (open) count_split<MODEL>(fits);
    fold();
    if (ONE) {  // the CTA adds its warps' sums up
        if (lane == 0) {
            sh.warp_fit[warp] = cur_chunks ? cur_fit : -1;
            sh.warp_chunks[warp] = cur_chunks;
        }
    } else if (cur_chunks) {
        flush_warp<MODEL>(sh.fit[0], cur_chunks, sh.pub[0][0]);
    }
}

template <int MODEL>
__device__ __noinline__ void run_wide_tiles(const FitDev* __restrict__ fits, const TileDev* __restrict__ tiles, int n_wide,
                                            const SplitDev* __restrict__ splits, unsigned* queue, int window_max, int cap,
                                            int* const status) {
    run_tiles<MODEL, false>(fits, tiles, 0, n_wide, splits, queue, window_max, cap, status);
}

// Tiles [0, n_wide) (windows that take a CTA's memory, or direct) are taken by
// whole CTAs, the rest by single warps.  cap: window entries a CTA's memory
// holds, at least narrow_cap() per warp and 8 more than the widest staged
// window.
template <int MODEL>
__global__ void __launch_bounds__(FUSED_THREADS, FUSED_MIN_CTAS)
em_fused_kernel(const FitDev* __restrict__ fits, const TileDev* __restrict__ tiles, int n_wide, int n_tiles,
                const SplitDev* __restrict__ splits, WorkState* ws, int window_max, int cap,
                const CountFitDev* __restrict__ cfits, int n_cfits, int count_blocks) {
    constexpr int NP = pub_slots(MODEL);
    extern __shared__ __align__(128) unsigned char smem[];
    Shared<MODEL>& sh = cta_shared<MODEL>();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n_warps = blockDim.x >> 5;
    int* const status = fits[0].status;
    static_assert(sizeof(FitDev) % 8 == 0 && sizeof(FitDev) <= 256, "FitDev is copied as 8-byte words, one per lane");
    static_assert(sizeof(TileDev) == 48 && sizeof(SplitDev) == 32, "copied in 16-byte units");

    for (int k = tid; k < n_warps * NP; k += blockDim.x) (&sh.wacc[0][0])[k] = 0.0;
    if (tid == 0) sh.abort = 0;
    if (n_wide) {
        run_wide_tiles<MODEL>(fits, tiles, n_wide, splits, &ws->next_tile[0], window_max, cap, status);
        __syncthreads();
    }
    if (!n_wide || *(volatile int*)&sh.abort == 0)
        run_tiles<MODEL, true>(fits, tiles, n_wide, n_tiles, splits, &ws->next_tile[1], window_max, cap, status);
    __syncthreads();
    if (warp == 0 && *(volatile int*)&sh.abort == 0) {
        // The warps' last sums, one flush per run of warps with the same fit
        // (usually all of them).
        for (int w = 0; w < n_warps;) {
            const int fit = sh.warp_fit[w];
            double v = 0.0, v2 = 0.0;
            unsigned chunks = 0;
            const float g = sh.pub[w][0];
            int e = w;
            for (; e < n_warps && sh.warp_fit[e] == fit; e++) {
                if (lane < NP) v += sh.wacc[e][lane];
                if (lane + 32 < NP) v2 += sh.wacc[e][lane + 32];
                chunks += sh.warp_chunks[e];
            }
            if (fit >= 0) flush_public(sh.fit[w], model_of<MODEL>(sh.fit[w]), lane, v, v2, g, chunks);
            w = e;
        }
    }

    // ---------------- count chunks of batched PBM / UBM fits ---------------
    // With the tile queue empty, the CTA takes chunks of kCountChunk pairs of
    // the batch's count-path fits from a second queue (count_step), in the
    // shared memory the tiles used: every tile's copies have been waited for,
    // and the last M-step ended before the barrier above.
    if (n_cfits > 0) {
        __shared__ int s_cchunk, s_cfit, s_cint[2];
        float* csm = reinterpret_cast<float*>(smem);
        for (;;) {
            __syncthreads();
            if (tid == 0) {
                const int c = *(volatile int*)&sh.abort ? count_blocks : (int)atomicAdd(&ws->next_count, 1u);
                s_cchunk = c;
                if (c < count_blocks) {  // the fit owning chunk c: last with blk_begin <= c
                    int lo = 0, hi = n_cfits - 1;
                    while (lo < hi) {
                        const int mid = (lo + hi + 1) / 2;
                        if (cfits[mid].blk_begin <= c) lo = mid; else hi = mid - 1;
                    }
                    s_cfit = lo;
                }
            }
            __syncthreads();
            const int c = s_cchunk;
            if (c >= count_blocks) break;
            const CountFitDev cf = cfits[s_cfit];
            const int64_t q0 = (int64_t)(c - cf.blk_begin) * kCountChunk;
            const int64_t q1 = q0 + kCountChunk < cf.n_qd ? q0 + kCountChunk : cf.n_qd;
            count_step<16, 4>(*cf.fit, cf.off, cf.ent, q0 + tid, q1, blockDim.x, (unsigned)cf.n_blocks, csm, s_cint);
        }
    }
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        unsigned e = atomicAdd(&ws->ctas_exited, 1u);
        if (e == gridDim.x - 1) {
            for (unsigned& q : ws->next_tile) q = 0;
            ws->next_count = 0;
            ws->ctas_exited = 0;
        }
    }
}

cudaError_t set_wait_hooks(unsigned long long wait_limit_ns, int stall_tile) {
    cudaError_t e = cudaMemcpyToSymbol(g_wait_limit_ns, &wait_limit_ns, sizeof wait_limit_ns);
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_stall_tile, &stall_tile, sizeof stall_tile);
    return e;
}

size_t fused_entry_bytes(int model) { return make_layout(model, 4).bytes / 4; }

int fused_narrow_cap(int model) { return narrow_cap(model); }

size_t fused_smem_bytes(int model, int cap, int warps, bool with_counts) {
    const size_t bytes = make_layout(model, cap).bytes + (size_t)warps * kChunkBytes;
    return with_counts && bytes < count_step_smem<16>() ? count_step_smem<16>() : bytes;
}

template <class F>
static auto with_kernel(int model, F&& go) {
    switch (model) {
        case PBM: return go(em_fused_kernel<PBM>);
        case CCM: return go(em_fused_kernel<CCM>);
        case DBN: return go(em_fused_kernel<DBN>);
        case UBM: return go(em_fused_kernel<UBM>);
        default: return go(em_fused_kernel<-1>);
    }
}

cudaError_t launch_em_fused(int model, const FitDev* fits, const TileDev* tiles, int n_wide, int n_tiles, const SplitDev* splits,
                            WorkState* ws, int window_max, int cap, int grid, int block, const CountFitDev* cfits,
                            int n_cfits, int count_blocks, cudaStream_t stream) {
    const size_t smem = fused_smem_bytes(model, cap, block / 32, n_cfits > 0);
    return with_kernel(model, [&](auto kernel) {
        kernel<<<grid, block, smem, stream>>>(fits, tiles, n_wide, n_tiles, splits, ws, window_max, cap, cfits, n_cfits, count_blocks);
        return cudaGetLastError();
    });
}

cudaError_t fused_set_smem_limit(int model, size_t bytes) {
    return with_kernel(model, [&](auto kernel) {
        return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    });
}

cudaError_t fused_static_smem(int model, size_t* bytes) {
    cudaFuncAttributes a{};
    const cudaError_t e = with_kernel(model, [&](auto kernel) { return cudaFuncGetAttributes(&a, kernel); });
    *bytes = a.sharedSizeBytes;
    return e;
}

cudaError_t fused_occupancy(int model, int block, size_t smem, int* blocks_per_sm) {
    return with_kernel(model, [&](auto kernel) {
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, kernel, block, smem);
    });
}

// Packs the tiles' sessions: per tile, chunks of 32 sessions, a chunk being
// five rows of 32 words (window positions of ranks 2j and 2j + 1 in the low
// and high half of row j's word) and 32 click masks (padding zeroed), so that
// the lanes of a warp read a chunk in six coalesced rows.  A position is the
// window entry itself or, slots = true, its byte offset in a slot of the EM
// kernel, 4 (entry + qd_begin % 4).  Sessions are
// ordered by click pattern (DBN: last-click rank; CCM: last-click rank, then
// mask; PBM/UBM: click mask) so the lanes of a warp take the same branches: a
// block radix sort of (pattern << 16 | position) on the pattern bits the
// model's E-step branches on, stable, so equal patterns keep their session
// order.  DBN and CCM sessions without clicks
// carry no variable statistic (their constant contributions are folded in at
// upload) and are left out: the host's s_packed counts those that remain.
// Direct tiles keep no packed block.
constexpr int kPackThreads = 256;
constexpr int kPackMinKeys = 4 * kPackThreads;  // keys[] holds at least this many

template <int ITEMS>
using PackSort = cub::BlockRadixSort<uint32_t, kPackThreads, ITEMS, cub::NullType, 5>;

union PackSortStorage {
    typename PackSort<4>::TempStorage s4;
    typename PackSort<8>::TempStorage s8;
    typename PackSort<16>::TempStorage s16;
};

// Sort keys of one tile's sessions, in blocked order (thread t holds
// positions t * ITEMS ...): pattern in the high half, position in the low;
// positions past the tile get the largest key.  Sorted keys go to keys[].
template <int ITEMS>
__device__ __forceinline__ void pack_sort(PackSortStorage& tmp, uint32_t* keys, const uint16_t* click, int64_t s_begin,
                                          int s_count, bool drop_clickless, int begin_bit) {
    uint32_t k[ITEMS];
#pragma unroll
    for (int j = 0; j < ITEMS; j++) {
        const int i = threadIdx.x * ITEMS + j;
        uint32_t key = 0xFFFFFFFFu;
        if (i < s_count) {
            const unsigned m = click[s_begin + i];
            const uint32_t k16 = drop_clickless ? (m ? (((uint32_t)(31 - __clz(m)) << 10) | m) : 0xFFFFu) : m;
            key = (k16 << 16) | (uint32_t)i;
        }
        k[j] = key;
    }
    // Patterns are below 0x2800; clickless sessions and padding (0xFFFF) read
    // 0x3FFF on bits [16, 30) and sort after them, padding last (stability).
    PackSort<ITEMS>(reinterpret_cast<typename PackSort<ITEMS>::TempStorage&>(tmp)).Sort(k, begin_bit, 30);
#pragma unroll
    for (int j = 0; j < ITEMS; j++) keys[threadIdx.x * ITEMS + j] = k[j];
}

// Three blocks per SM (80 registers): 0.2 ms less per upload of 16M sessions
// than two blocks at the 116 registers the 16-item sort would take.
__global__ void __launch_bounds__(kPackThreads, 3) pack_tiles_kernel(int model, TileDev* tiles, int n_tiles, int window_max,
                                                                 const int32_t* planes, int64_t stride,
                                                                 const uint16_t* click, unsigned char* tblk, int* status, bool slots) {
    extern __shared__ uint32_t keys[];   // sort keys
    __shared__ PackSortStorage sort_tmp;
    __shared__ int s_kept;
    for (int t = blockIdx.x; t < n_tiles; t += gridDim.x) {
        const TileDev tile = tiles[t];
        if (tile.qd_count > window_max) continue;
        const bool drop_clickless = model == DBN || model == CCM;
        // The DBN E-step branches on the last-click rank only: one radix pass
        // over its 4 bits; CCM also on the clicks before it, PBM / UBM on the
        // mask: the 14 pattern bits.
        const int begin_bit = model == DBN ? 26 : 16;
        if (tile.s_count <= 4 * kPackThreads)
            pack_sort<4>(sort_tmp, keys, click, tile.s_begin, tile.s_count, drop_clickless, begin_bit);
        else if (tile.s_count <= 8 * kPackThreads)
            pack_sort<8>(sort_tmp, keys, click, tile.s_begin, tile.s_count, drop_clickless, begin_bit);
        else
            pack_sort<16>(sort_tmp, keys, click, tile.s_begin, tile.s_count, drop_clickless, begin_bit);
        __syncthreads();
        int kept = 0;
        for (int i = threadIdx.x; i < tile.s_count; i += blockDim.x) kept += (keys[i] >> 16) != 0xFFFFu;
        if (threadIdx.x == 0) s_kept = 0;
        __syncthreads();
        atomicAdd(&s_kept, kept);
        __syncthreads();
        // The host sized the tile's block for tile.s_packed sessions.
        if (s_kept != tile.s_packed && threadIdx.x == 0) atomicOr(status, ST_BAD_INDEX);
        const int n_kept = min(s_kept, tile.s_packed);
        const uint32_t pos0 = slots ? (uint32_t)(tile.qd_begin & 3) : 0u;
        const int pos_shift = slots ? 2 : 0;
        for (int i = threadIdx.x; i < ((tile.s_packed + 31) & ~31); i += blockDim.x) {
            const bool in = i < n_kept;
            const int64_t s = tile.s_begin + (in ? (int64_t)(keys[i] & 0xFFFFu) : 0);
            unsigned char* const chunk = tblk + tile.blk_off + (int64_t)(i >> 5) * kChunkBytes;
            // The ten gathers of a session are under way together (one pair of
            // ranks after another took 1.35 ms at 16M sessions, this 0.66).
            int v[MC_R];
#pragma unroll
            for (int r = 0; r < MC_R; r++) v[r] = in ? __ldg(planes + (int64_t)r * stride + s) : 0;
            const uint16_t m = in ? click[s] : (uint16_t)0;
            bool bad = false;
#pragma unroll
            for (int j = 0; j < MC_R / 2; j++) {
                uint32_t w = 0;
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    int64_t p = in ? (int64_t)v[2 * j + h] - tile.qd_begin : 0;
                    if (p < 0 || p >= tile.qd_count) { bad = true; p = 0; }
                    w |= (((uint32_t)p + pos0) << pos_shift) << (16 * h);
                }
                reinterpret_cast<uint32_t*>(chunk)[j * 32 + (i & 31)] = w;
            }
            if (bad) atomicOr(status, ST_BAD_INDEX);
            reinterpret_cast<uint16_t*>(chunk + 5 * 128)[i & 31] = m;
        }
        __syncthreads();
    }
}

// Blocks' largest packed occurrence counts (sessions with a click for DBN and
// CCM, else all): a CTA per block, the window's counts in shared memory.
__global__ void __launch_bounds__(256) block_occ_kernel(int model, const TileDev* __restrict__ blocks, int n_blocks, int window_max,
                                                        const int32_t* __restrict__ planes, int64_t stride,
                                                        const uint16_t* __restrict__ click, int* __restrict__ occ) {
    extern __shared__ unsigned cnt[];
    __shared__ int s_max;
    for (int b = blockIdx.x; b < n_blocks; b += gridDim.x) {
        const TileDev blk = blocks[b];
        if (blk.qd_count > window_max) continue;
        __syncthreads();
        for (int i = threadIdx.x; i < blk.qd_count; i += blockDim.x) cnt[i] = 0;
        if (threadIdx.x == 0) s_max = 0;
        __syncthreads();
        for (int i = threadIdx.x; i < blk.s_count; i += blockDim.x) {
            const int64_t s = blk.s_begin + i;
            if ((model == DBN || model == CCM) && click[s] == 0) continue;
            for (int r = 0; r < MC_R; r++) {
                const int64_t p = (int64_t)planes[(int64_t)r * stride + s] - blk.qd_begin;
                if (p >= 0 && p < blk.qd_count) atomicAdd(cnt + p, 1u);
            }
        }
        __syncthreads();
        unsigned mx = 0;
        for (int i = threadIdx.x; i < blk.qd_count; i += blockDim.x) mx = max(mx, cnt[i]);
        mx = __reduce_max_sync(FULL_MASK, mx);
        if ((threadIdx.x & 31) == 0 && mx) atomicMax(&s_max, (int)mx);
        __syncthreads();
        if (threadIdx.x == 0) occ[b] = s_max;
    }
}

__global__ void tile_occ_kernel(TileDev* tiles, int n_tiles, const int* __restrict__ occ) {
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n_tiles; t += gridDim.x * blockDim.x) tiles[t].max_occ = occ[tiles[t].max_occ];
}

cudaError_t launch_block_occ(int model, const TileDev* blocks, int n_blocks, int window_max, const int32_t* planes, int64_t stride,
                             const uint16_t* click, int* occ, int n_sm, cudaStream_t st) {
    if (n_blocks == 0) return cudaSuccess;
    const size_t smem = (size_t)window_max * 4;
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(block_occ_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    block_occ_kernel<<<n_blocks < 8 * n_sm ? n_blocks : 8 * n_sm, 256, smem, st>>>(model, blocks, n_blocks, window_max, planes, stride,
                                                                                  click, occ);
    return cudaGetLastError();
}

cudaError_t launch_tile_occ(TileDev* tiles, int n_tiles, const int* occ, int n_sm, cudaStream_t st) {
    if (n_tiles == 0) return cudaSuccess;
    const int g = (n_tiles + 255) / 256;
    tile_occ_kernel<<<g < 8 * n_sm ? g : 8 * n_sm, 256, 0, st>>>(tiles, n_tiles, occ);
    return cudaGetLastError();
}

cudaError_t launch_pack_tiles(int model, TileDev* tiles, int n_tiles, int window_max, int max_tile_sessions, const int32_t* planes,
                              int64_t stride, const uint16_t* click, unsigned char* tblk, int* status, bool slots,
                              int n_sm, cudaStream_t st) {
    if (n_tiles == 0) return cudaSuccess;
    // keys[] holds 256 x ITEMS keys of the largest class a tile may take.
    int P = kPackMinKeys;
    while (P < max_tile_sessions) P <<= 1;
    int g = n_tiles < 8 * n_sm ? n_tiles : 8 * n_sm;
    const size_t smem = (size_t)P * 4;
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(pack_tiles_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    pack_tiles_kernel<<<g, kPackThreads, smem, st>>>(model, tiles, n_tiles, window_max, planes, stride, click, tblk,
                                                     status, slots);
    return cudaGetLastError();
}

}  // namespace mcd
