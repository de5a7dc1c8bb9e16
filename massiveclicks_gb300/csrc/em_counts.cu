// PBM and UBM EM iterations from counts per (qd, statistic key).
//
// In the PBM and UBM E-steps (pbm.cu:191-253, ubm.cu:185-247) an unclicked
// occurrence of pair qd under examination parameter e_k adds
// (a - a e_k) / (1 - a e_k) to the qd's attractiveness numerator and, unless
// a later rank of the same session writes the same UBM slot (last write wins),
// (e_k - a e_k) / (1 - a e_k) to parameter k's numerator; a clicked occurrence
// adds constants (folded into the fit's constants at upload).  The key k is
// the rank (PBM) or the examination slot r(r+1)/2 + previous click (UBM), so
// the terms depend on the session only through (qd, k, alive) and
//   numerator of qd = clicks + sum over entries count * f(a_qd, e_k)
//   numerator of k  = constants + sum over alive entries count * h(a_qd, e_k).
// At upload every unclicked occurrence becomes a 64-bit key (qd, k, alive);
// sorting and run-length encoding them gives the entries of each qd (CSR).
// An iteration is one pass over the qd pairs: a thread takes a qd, evaluates
// its entries and runs its M-step in place.  The public terms go into
// per-warp shared bins (dense PBM kernel: registers), then block sums (as
// integers, count_step.cuh; dense: FP64), then one FP64 global atomic per
// parameter per block, into one of eight copies of the fit's bins (dense: one);
// the block that finishes last runs the public M-step into the other half of
// the double buffer, as the tile kernel does, so the fit's state (pub_theta,
// iter) is the same for both paths.
#include <cstdint>
#include <cuda_runtime.h>
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_run_length_encode.cuh>
#include <cub/device/device_scan.cuh>
#include <thrust/iterator/reverse_iterator.h>

#include "common.cuh"
#include "count_step.cuh"
#include "devmem.h"
#include "kernels.h"

namespace mcd {

constexpr uint32_t kMaxCount = 1u << 25;  // count field of an entry

// Keys ((qd << 7) | (k << 1) | alive) of the unclicked occurrences; a clicked
// occurrence gets the all-ones key, which sorts after every real key.  The key
// of (session s, rank r) sits at r * n + s: the sort does not care where a key
// starts, and rank-major positions make the stores coalesced.
template <class K>
__global__ void count_keys_kernel(int64_t n, int64_t stride, const int32_t* __restrict__ planes,
                                  const uint16_t* __restrict__ click, int model, K* __restrict__ keys) {
    const int64_t step = (int64_t)gridDim.x * blockDim.x;
    for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < n; s += step) {
        const unsigned m = click[s];
        int slot[MC_R];
        int last = 9;
#pragma unroll
        for (int r = 0; r < MC_R; r++) {
            slot[r] = model == PBM ? r : r * (r + 1) / 2 + last;
            if ((m >> r) & 1u) last = r;
        }
#pragma unroll
        for (int r = 0; r < MC_R; r++) {
            K key = ~K(0);
            if (!((m >> r) & 1u)) {
                bool alive = true;
#pragma unroll
                for (int r2 = r + 1; r2 < MC_R; r2++) alive = alive && slot[r2] != slot[r];
                const K p = (K)planes[(int64_t)r * stride + s];
                key = (p << 7) | ((K)slot[r] << 1) | (alive ? K(1) : K(0));
            }
            keys[(int64_t)r * n + s] = key;
        }
    }
}

// Entry i = (count << 7) | (k << 1) | alive of run i; flags a count too large.
template <class K>
__global__ void count_entries_kernel(int64_t runs, const K* __restrict__ uniq, const uint32_t* __restrict__ counts,
                                     uint32_t* __restrict__ ent, int* overflow) {
    const int64_t step = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < runs; i += step) {
        const uint32_t c = counts[i];
        if (c >= kMaxCount) atomicOr(overflow, 1);
        ent[i] = (c << 7) | (uint32_t)(uniq[i] & K(0x7F));
    }
}

// off[q] = first run whose qd is >= q, for q in [0, n_qd], in two parallel
// steps: the first run of each qd writes its index at off[qd] (the others
// hold ~0, off[n_qd] = runs), then a suffix minimum fills each gap with the
// next qd's value.
template <class K>
__global__ void count_first_run_kernel(int64_t runs, const K* __restrict__ uniq, uint32_t* __restrict__ off) {
    const int64_t step = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < runs; i += step) {
        const int64_t q = (int64_t)(uniq[i] >> 7);
        if (i == 0 || (int64_t)(uniq[i - 1] >> 7) != q) off[q] = (uint32_t)i;
    }
}

struct MinU32 {
    __device__ __forceinline__ uint32_t operator()(uint32_t a, uint32_t b) const { return a < b ? a : b; }
};

// PBM: a warp per chunk of 32 qd packs its counts and clicks (see the kernel),
// the wide chunks numbered by *n_wide, and with `wide` writes those; flags a
// count above 65535.
template <class K>
__global__ void __launch_bounds__(256) count_dense_kernel(int64_t n_qd, const K* __restrict__ uniq, const uint32_t* __restrict__ counts,
                                                          const uint32_t* __restrict__ off, const uint2* __restrict__ cnt,
                                                          uint32_t* __restrict__ rows, uint32_t* __restrict__ wide, int* n_wide,
                                                          int* overflow) {
    const int lane = threadIdx.x & 31;
    const int64_t chunks = (n_qd + 31) >> 5;
    for (int64_t c = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5); c < chunks; c += (int64_t)gridDim.x * 8) {
        uint32_t* const p = rows + c * 96 + lane;
        if (wide && p[64] != 0xFFFFFFFFu) continue;
        const int64_t q = c * 32 + lane;
        uint32_t k[MC_R] = {};
        uint32_t clicks = 0, most = 0;
        if (q < n_qd) {
            clicks = cnt[q].y;
            for (uint32_t i = off[q]; i < off[q + 1]; i++) {
                const uint32_t n = counts[i];
                const int r = (int)((uniq[i] >> 1) & K(63));
                most = max(most, n);
#pragma unroll
                for (int j = 0; j < MC_R; j++)
                    if (j == r) k[j] = n;
            }
        }
        if (wide) {
            uint32_t* const to = wide + (int64_t)p[0] * 160 + lane;
#pragma unroll
            for (int j = 0; j < MC_R / 2; j++) to[j * 32] = k[2 * j] | k[2 * j + 1] << 16;
            continue;
        }
        if (most > 0xFFFFu) atomicOr(overflow, 1);
        if (__any_sync(0xffffffffu, most > 0xFFu || clicks > 0xFFFEu)) {
            int at = lane == 0 ? atomicAdd(n_wide, 1) : 0;
            at = __shfl_sync(0xffffffffu, at, 0);
            p[0] = (uint32_t)at;
            p[32] = 0u;
            p[64] = 0xFFFFFFFFu;
        } else {
            p[0] = k[0] | k[1] << 8 | k[2] << 16 | k[3] << 24;
            p[32] = k[4] | k[5] << 8 | k[6] << 16 | k[7] << 24;
            p[64] = k[8] | k[9] << 8 | clicks << 16;
        }
    }
}

static int grid_for(int64_t n, int n_sm) {
    int64_t b = (n + 255) / 256;
    int g = (int)(b < 16 * n_sm ? b : 16 * n_sm);
    return g < 1 ? 1 : g;
}

template <class T>
static cudaError_t tmp_alloc(T** p, size_t count) {
    return mch::dev_alloc(reinterpret_cast<void**>(p), count * sizeof(T) > 0 ? count * sizeof(T) : 1);
}

// K = uint32_t while qd < 2^25 - 1 (the all-ones key stays above every real
// key), else uint64_t.  The sort runs over the low end_bit bits, the fewest
// that hold every real key below 2^end_bit - 1.
template <class K>
static cudaError_t build_counts_t(int model, int64_t n, int64_t stride, int64_t n_qd, const int32_t* planes,
                                  const uint16_t* click, const uint2* cnt, int n_sm, cudaStream_t st, uint32_t** off_out,
                                  uint32_t** ent_out, int64_t* n_entries, DenseTable* dense_out, int* usable) {
    const int64_t nk = n * MC_R;
    K *keys = nullptr, *alt = nullptr;
    uint32_t* counts = nullptr;
    int64_t* d_small = nullptr;  // [0] run count, [1] overflow flags: CSR (low word), dense (high word), [2] wide chunks
    void* temp = nullptr;
    uint32_t *off = nullptr, *ent = nullptr;
    uint32_t *rows = nullptr, *wide = nullptr;
    cudaError_t e = cudaSuccess;
    auto ck = [&](cudaError_t x) { if (e == cudaSuccess) e = x; };
    auto release = [&]() {  // after the stream has drained
        cudaStreamSynchronize(st);
        mch::dev_free(keys); mch::dev_free(alt); mch::dev_free(counts); mch::dev_free(d_small); mch::dev_free(temp);
    };
    int end_bit = 8;
    while (end_bit < (int)(8 * sizeof(K)) && (((int64_t)1 << (end_bit - 7)) - 1) < n_qd) end_bit++;
    ck(tmp_alloc(&keys, (size_t)nk));
    ck(tmp_alloc(&alt, (size_t)nk));
    ck(tmp_alloc(&counts, (size_t)nk));
    ck(tmp_alloc(&d_small, 3));
    size_t sort_bytes = 0, rle_bytes = 0;
    cub::DoubleBuffer<K> db(keys, alt);
    if (e == cudaSuccess) {
        ck(cub::DeviceRadixSort::SortKeys(nullptr, sort_bytes, db, (int64_t)nk, 0, end_bit, st));
        ck(cub::DeviceRunLengthEncode::Encode(nullptr, rle_bytes, keys, alt, counts, d_small, (int64_t)nk, st));
        ck(mch::dev_alloc(&temp, sort_bytes > rle_bytes ? sort_bytes : rle_bytes));
    }
    if (e != cudaSuccess) { release(); return e; }
    ck(cudaMemsetAsync(d_small, 0, 24, st));
    count_keys_kernel<K><<<grid_for(n, n_sm), 256, 0, st>>>(n, stride, planes, click, model, keys);
    ck(cudaGetLastError());
    ck(cub::DeviceRadixSort::SortKeys(temp, sort_bytes, db, (int64_t)nk, 0, end_bit, st));
    K* sorted = db.Current();
    K* uniq = db.Alternate();
    ck(cub::DeviceRunLengthEncode::Encode(temp, rle_bytes, sorted, uniq, counts, d_small, (int64_t)nk, st));
    int64_t runs = 0;
    ck(cudaMemcpyAsync(&runs, d_small, 8, cudaMemcpyDeviceToHost, st));
    ck(cudaStreamSynchronize(st));
    if (e != cudaSuccess) { release(); return e; }
    // The clicked occurrences form the last run (the all-ones key), if any.
    if (runs > 0) {
        K last_key = 0;
        ck(cudaMemcpy(&last_key, uniq + runs - 1, sizeof(K), cudaMemcpyDeviceToHost));
        if (last_key == ~K(0)) runs--;
    }
    const uint32_t runs32 = (uint32_t)runs;  // < 2^32: n * 10 < 2^32 entries at most
    ck(tmp_alloc(&off, (size_t)n_qd + 1));
    ck(tmp_alloc(&ent, (size_t)(runs > 0 ? runs : 1)));
    if (model == PBM && dense_out) ck(tmp_alloc(&rows, (size_t)((n_qd + 31) >> 5) * 96));
    int* overflow = reinterpret_cast<int*>(d_small + 1);
    if (e == cudaSuccess) {
        ck(cudaMemsetAsync(off, 0xFF, (size_t)n_qd * sizeof(uint32_t), st));
        ck(cudaMemcpyAsync(off + n_qd, &runs32, sizeof(uint32_t), cudaMemcpyHostToDevice, st));
        count_entries_kernel<K><<<grid_for(runs, n_sm), 256, 0, st>>>(runs, uniq, counts, ent, overflow);
        ck(cudaGetLastError());
        count_first_run_kernel<K><<<grid_for(runs, n_sm), 256, 0, st>>>(runs, uniq, off);
        ck(cudaGetLastError());
        {
            auto rev = thrust::make_reverse_iterator(off + n_qd + 1);
            size_t scan_bytes = 0;
            ck(cub::DeviceScan::InclusiveScan(nullptr, scan_bytes, rev, rev, MinU32(), (int64_t)n_qd + 1, st));
            void* scan_tmp = nullptr;
            ck(mch::dev_alloc(&scan_tmp, scan_bytes ? scan_bytes : 1));
            if (e == cudaSuccess)
                ck(cub::DeviceScan::InclusiveScan(scan_tmp, scan_bytes, rev, rev, MinU32(), (int64_t)n_qd + 1, st));
            if (scan_tmp) {
                cudaStreamSynchronize(st);
                mch::dev_free(scan_tmp);
            }
        }
        if (rows) {
            count_dense_kernel<K><<<grid_for(n_qd, n_sm), 256, 0, st>>>(n_qd, uniq, counts, off, cnt, rows, nullptr, overflow + 2,
                                                                        overflow + 1);
            ck(cudaGetLastError());
        }
    }
    int flags[3] = {0, 0, 0};
    ck(cudaMemcpyAsync(flags, overflow, 12, cudaMemcpyDeviceToHost, st));
    ck(cudaStreamSynchronize(st));
    if (e == cudaSuccess && rows && !flags[0] && !flags[1] && flags[2]) {
        ck(tmp_alloc(&wide, (size_t)flags[2] * 160));
        if (e == cudaSuccess) {
            count_dense_kernel<K><<<grid_for(n_qd, n_sm), 256, 0, st>>>(n_qd, uniq, counts, off, cnt, rows, wide, nullptr, nullptr);
            ck(cudaGetLastError());
        }
    }
    release();
    if (e != cudaSuccess || flags[0]) {
        mch::dev_free(off);
        mch::dev_free(ent);
        mch::dev_free(rows);
        mch::dev_free(wide);
        return e;  // on overflow: success without the count path
    }
    if (flags[1]) {  // a count above 16 bits: the entries only
        mch::dev_free(rows);
        rows = nullptr;
    }
    *off_out = off;
    *ent_out = ent;
    *n_entries = runs;
    if (dense_out) *dense_out = DenseTable{rows, wide, flags[2]};
    *usable = 1;
    return cudaSuccess;
}

void free_dense(DenseTable* t) {
    mch::dev_free(const_cast<uint32_t*>(t->rows));
    mch::dev_free(const_cast<uint32_t*>(t->wide));
    *t = DenseTable{};
}

int64_t dense_table_bytes(const DenseTable& t, int64_t n_qd) {
    return t.rows ? (int64_t)sizeof(uint32_t) * (((n_qd + 31) >> 5) * 96 + (int64_t)t.n_wide * 160) : 0;
}

cudaError_t build_counts(int model, int64_t n, int64_t stride, int64_t n_qd, const int32_t* planes, const uint16_t* click,
                         const uint2* cnt, int n_sm, cudaStream_t st, uint32_t** off_out, uint32_t** ent_out, int64_t* n_entries,
                         DenseTable* dense_out, int* usable) {
    *off_out = nullptr;
    *ent_out = nullptr;
    *n_entries = 0;
    if (dense_out) *dense_out = DenseTable{};
    *usable = 0;
    if (n * MC_R >= ((int64_t)1 << 32) || n_qd >= ((int64_t)1 << 56)) return cudaSuccess;  // keep the tile path
    if (n_qd <= ((int64_t)1 << 25) - 2)
        return build_counts_t<uint32_t>(model, n, stride, n_qd, planes, click, cnt, n_sm, st, off_out, ent_out, n_entries,
                                        dense_out, usable);
    return build_counts_t<unsigned long long>(model, n, stride, n_qd, planes, click, cnt, n_sm, st, off_out, ent_out, n_entries,
                                              dense_out, usable);
}

// One thread per qd: its entries, its M-step in place; the public terms of the
// alive entries go into per-warp shared bins.  Bound by the latency of a pair's
// entries, one after another, and by lane divergence: 64 warps per SM at 32
// registers hide more of it than prefetches at 40 do (16M UBM sessions: 241 us
// per iteration then, 291 with the next two pairs read ahead), and bins of every
// lane's own in place of atomics leave 28 warps (240 us, with other rounding).
// A warp per 32 qd with coalesced entry reads, and pairs sorted by their
// entries, were slower too.
//
// One block's share of an iteration: count_step (count_step.cuh) over static
// shared memory.
template <int COPIES, int UNROLL>
__device__ __forceinline__ void count_iteration(const FitDev& f, const uint32_t* __restrict__ off,
                                                const uint32_t* __restrict__ ent, int64_t q_first, int64_t q_end,
                                                int64_t q_step, unsigned n_blocks) {
    __shared__ __align__(16) float sm[count_step_smem<COPIES>() / sizeof(float)];
    __shared__ int s_int[2];
    count_step<COPIES, UNROLL>(f, off, ent, q_first, q_end, q_step, n_blocks, sm, s_int);
}

// One fit: blocks stride over its qd.
template <int COPIES>
__global__ void __launch_bounds__(256, 8) em_counts_kernel(const FitDev* __restrict__ fp, const uint32_t* __restrict__ off,
                                                        const uint32_t* __restrict__ ent) {
    const FitDev& f = *fp;
    count_iteration<COPIES, 1>(f, off, ent, (int64_t)blockIdx.x * blockDim.x + threadIdx.x, f.n_qd,
                            (int64_t)gridDim.x * blockDim.x, gridDim.x);
}

// Grid of a grid-stride count launch: enough blocks for one qd per thread, at
// most blocks_per_sm per SM.
static int count_grid(int64_t n_qd, int block, int blocks_per_sm, int n_sm) {
    const int64_t blocks = (n_qd + block - 1) / block;
    const int64_t cap = (int64_t)blocks_per_sm * n_sm;
    const int g = (int)(blocks < cap ? blocks : cap);
    return g < 1 ? 1 : g;
}

bool count_shape_valid(const CountShape& c, bool dense) {
    if (c.block < 64 || c.block > 256 || c.block % 32 || c.blocks_per_sm < 1 || c.blocks_per_sm > 32) return false;
    return dense || c.copies == 4 || c.copies == 8 || c.copies == 16;
}

cudaError_t launch_em_counts(const FitDev* fit, const uint32_t* off, const uint32_t* ent, int64_t n_qd, int n_sm,
                             const CountShape& c, cudaStream_t st) {
    const int g = count_grid(n_qd, c.block, c.blocks_per_sm, n_sm);
    switch (c.copies) {
        case 4: em_counts_kernel<4><<<g, c.block, 0, st>>>(fit, off, ent); break;
        case 16: em_counts_kernel<16><<<g, c.block, 0, st>>>(fit, off, ent); break;
        default: em_counts_kernel<8><<<g, c.block, 0, st>>>(fit, off, ent); break;
    }
    return cudaGetLastError();
}

// Pairs of FP32 operations in one instruction each (PTX ISA: .f32x2), rounded as
// the single ones.
struct F2 {
    unsigned long long v;
};
__device__ __forceinline__ F2 pack2(float x, float y) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float2 unpack2(F2 a) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a.v));
    return r;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}

__device__ __forceinline__ F2 add2(F2 a, F2 b) {
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
// Bytes i and i + 1 of w as floats: 2^23 + byte is the byte below the exponent of
// 2^23 (a conversion takes a slot of the reciprocals' unit).
__device__ __forceinline__ F2 bytes2(uint32_t w, int i) {
    const float x = __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440u + i));
    const float y = __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7441u + i));
    return add2(pack2(x, y), pack2(-8388608.0f, -8388608.0f));
}

// PBM from dense counts: the unclicked occurrences of a qd at ranks 0..9, so
// every thread runs the same ten-rank loop and the rank sums stay in registers
// (no shared atomics); warp sums, then FP64 block sums, then one global atomic
// per rank per block.  A chunk of 32 qd has three words per qd, a plane of 32
// each: ranks 0..3 and 4..7 in bytes, ranks 8 and 9 in bytes and the clicks in
// 16 bits.  A chunk with larger counts has its index among the wide chunks in
// the first word, all ones in the third, and five words of two 16-bit counts
// per qd in the wide table.
//
// Bound by instruction issue and the reciprocals' unit (ten of them and about 130
// other operations per qd) near the memory's time: 20 bytes per qd and
// iteration.  16-bit rows of 20 bytes, scalar operations and exact occurrence
// counts beside them (36 bytes) took 207 us per iteration at 22.6M qd (16M
// sessions), this 123; 24 and 17 us at 1.2M qd, 7.4 and 6.0 at 32k sessions.
//
// The qd of a virtual block are those that it would take of a grid-stride grid
// of `grid` blocks, and the FP32 sums are a virtual warp's.  A block is one
// virtual block, or with `shared` eight warps take twelve virtual warps: warp w
// < 4 the first half of a third one and then one, warp w + 4 one and then, with
// the sums so far handed over, the second half of the third.  Six blocks per SM
// sum as before and four run at a time, each as long.
template <bool SHARED>
__global__ void __launch_bounds__(256, 4) em_counts_pbm_dense_kernel(const FitDev* __restrict__ fp, DenseTable t, int grid) {
    __shared__ float wsum[SHARED ? 12 : 8][MC_R];  // of the virtual warps
    __shared__ float2 e[MC_R / 2];
    __shared__ float handed[SHARED ? 4 : 1][MC_R][32];
    __shared__ int s_it;
    const FitDev& f = *fp;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t n_qd = f.n_qd;
    const int64_t step = (int64_t)grid * blockDim.x;
    const int64_t half = (n_qd / step + 1) / 2 * step;
    // The qd of virtual warp v: first + v * 32, + step, ... in [first, end).
    auto virtual_warp = [&](int w) { return ((int64_t)blockIdx.x * (SHARED ? 12 : blockDim.x / 32) + w) * 32 + lane; };
    int64_t q = virtual_warp(SHARED && warp < 4 ? 8 + warp : warp);
    int64_t end = SHARED && warp < 4 ? min(q + half, n_qd) : n_qd;
    // A qd's words and value are read two passes ahead.
    struct Row {
        uint32_t w0, w1, w2;
        float a;
    };
    auto row = [&](int64_t at) {
        Row r{0u, 0u, 0u, 0.0f};
        if (at >= end) return r;
        const uint32_t* p = t.rows + (at >> 5) * 96 + lane;
        asm volatile("ld.global.nc.L1::no_allocate.b32 %0, [%1];" : "=r"(r.w0) : "l"(p));
        asm volatile("ld.global.nc.L1::no_allocate.b32 %0, [%1];" : "=r"(r.w1) : "l"(p + 32));
        asm volatile("ld.global.nc.L1::no_allocate.b32 %0, [%1];" : "=r"(r.w2) : "l"(p + 64));
        asm volatile("ld.global.L1::no_allocate.f32 %0, [%1];" : "=f"(r.a) : "l"(f.atr + at));
        return r;
    };
    Row r = row(q), next = row(q + step);
    if (tid == 0) s_it = *(volatile int*)f.iter;
    __syncthreads();
    if (tid < MC_R) reinterpret_cast<float*>(e)[tid] = f.pub_theta[(s_it & 1) * MC_MAX_PUB + tid];
    __syncthreads();
    F2 acc[MC_R / 2], ee[MC_R / 2];
#pragma unroll
    for (int j = 0; j < MC_R / 2; j++) {
        acc[j] = pack2(0.0f, 0.0f);
        ee[j] = pack2(e[j].x, e[j].y);
    }
    const F2 one = pack2(1.0f, 1.0f);
    // Values below `bound` (as bits: 1 while every examination is in [0, 1], as
    // the M-step leaves them) have 1 - a e in [2^-24, 1] at every rank, and a
    // rank without occurrences adds 0 times a finite value.  Values that a caller
    // has set otherwise leave the ranks without occurrences out one by one.
    uint32_t bound = 0x3F800000u;
#pragma unroll
    for (int j = 0; j < MC_R / 2; j++)
        if (!(e[j].x >= 0.0f && e[j].x <= 1.0f && e[j].y >= 0.0f && e[j].y <= 1.0f)) bound = 0u;
    for (int part = 0;; part++) {
        for (; q < end; q += step) {
            const Row after = row(q + 2 * step);
            const float a = r.a;
            const F2 aa = pack2(a, a), na = pack2(-a, -a);
            float v0 = 0.0f;
            // Ranks 2 j and 2 j + 1 with counts k.
            auto ranks = [&](int j, F2 k) {
                const float2 y = unpack2(fma2(na, ee[j], one));  // 1 - a e
                const F2 w = mul2(k, pack2(reciprocal(y.x), reciprocal(y.y)));
                const float2 d = unpack2(fma2(na, ee[j], aa)), ws = unpack2(w);
                v0 = __fmaf_rn(ws.x, d.x, v0);
                v0 = __fmaf_rn(ws.y, d.y, v0);
                acc[j] = fma2(w, fma2(na, ee[j], ee[j]), acc[j]);
            };
            uint2 n;
            if (r.w2 != 0xFFFFFFFFu && __float_as_uint(a) < bound) {
                ranks(0, bytes2(r.w0, 0));
                ranks(1, bytes2(r.w0, 2));
                ranks(2, bytes2(r.w1, 0));
                ranks(3, bytes2(r.w1, 2));
                ranks(4, bytes2(r.w2, 0));
                n.y = r.w2 >> 16;
                n.x = __dp4a(r.w0, 0x01010101u, __dp4a(r.w1, 0x01010101u, __dp4a(r.w2, 0x00000101u, n.y)));
            } else {
                const uint32_t* p = t.wide + (int64_t)r.w0 * 160 + lane;
                const bool wide = r.w2 == 0xFFFFFFFFu;
                n = f.cnt[q];
                if (__float_as_uint(a) < bound) {
#pragma unroll
                    for (int j = 0; j < MC_R / 2; j++) {
                        const uint32_t k = __ldg(p + j * 32);
                        ranks(j, pack2((float)(k & 0xFFFFu), (float)(k >> 16)));
                    }
                } else {
                    auto term = [&](float k, float x, float& sum) {
                        if (k == 0.0f) return;
                        const float w = k * __fdividef(1.0f, __fmaf_rn(-a, x, 1.0f));
                        v0 = __fmaf_rn(w, __fmaf_rn(-a, x, a), v0);
                        sum = __fmaf_rn(w, __fmaf_rn(-a, x, x), sum);
                    };
#pragma unroll
                    for (int j = 0; j < MC_R / 2; j++) {
                        const uint32_t b = (j < 2 ? r.w0 : j < 4 ? r.w1 : r.w2) >> 16 * (j & 1);
                        const uint32_t k = wide ? __ldg(p + j * 32) : (b & 0xFFu) | (b & 0xFF00u) << 8;
                        const float2 x = unpack2(ee[j]);
                        float2 sum = unpack2(acc[j]);
                        term((float)(k & 0xFFFFu), x.x, sum.x);
                        term((float)(k >> 16), x.y, sum.y);
                        acc[j] = pack2(sum.x, sum.y);
                    }
                }
            }
            const float v = __fdividef(1.0f + (float)n.y + v0, 2.0f + (float)n.x);
            f.atr[q] = v < MC_TOP ? v : MC_TOP;
            r = next;
            next = after;
        }
        __syncwarp();
        const bool hand = SHARED && part == 0 && warp < 4;
        if (SHARED && part == 0) {  // the other part's first rows
            const int64_t third = virtual_warp(8 + (warp & 3));
            q = warp < 4 ? virtual_warp(warp) : third + half;
            end = n_qd;
            r = row(q);
            next = row(q + step);
        }
#pragma unroll
        for (int j = 0; j < MC_R; j++) {
            const float2 both = unpack2(acc[j / 2]);
            float v = j & 1 ? both.y : both.x;
            if (hand) {
                handed[warp & 3][j][lane] = v;
                continue;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0) wsum[SHARED && part == 1 ? (warp < 4 ? warp : warp + 4) : warp][j] = v;
        }
        if (!SHARED || part == 1) break;
        // Barrier 1 + w of the two warps: the first arrives, the second waits.
        if (hand) {
            __threadfence_block();
            asm volatile("bar.arrive %0, 64;" ::"r"(1 + (warp & 3)) : "memory");
#pragma unroll
            for (int j = 0; j < MC_R / 2; j++) acc[j] = pack2(0.0f, 0.0f);
        } else {
            asm volatile("bar.sync %0, 64;" ::"r"(1 + (warp & 3)) : "memory");
#pragma unroll
            for (int j = 0; j < MC_R / 2; j++) acc[j] = pack2(handed[warp & 3][2 * j][lane], handed[warp & 3][2 * j + 1][lane]);
        }
    }
    __syncthreads();
    if (tid < MC_R) {
        double s = 0.0;
        for (int w = 0; w < (SHARED ? 12 : (int)(blockDim.x >> 5)); w++) s += (double)wsum[w][tid];
        if (s != 0.0) atomicAdd(f.pub_bins + 2 * tid, s);
    }
    __shared__ int s_last;
    count_public_finish<1>(f, s_it, gridDim.x, &s_last);
}

cudaError_t launch_em_counts_pbm_dense(const FitDev* fit, const DenseTable& dense, int64_t n_qd, int n_sm,
                                       const CountShape& c, cudaStream_t st) {
    const int grid = count_grid(n_qd, c.block, c.blocks_per_sm, n_sm);
    // Six blocks per SM, of which four run at a time: 22.6M qd took 145 us per
    // iteration one after another, 123 as four that share their qd; 11.3M 75 and
    // 68.5; 5.6M (24 qd per thread) 40.4 and 40.9, 1.2M 17.0 and 19.4.
    if (c.block == 256 && grid == 6 * n_sm && n_qd >= 32 * (int64_t)256 * grid)
        em_counts_pbm_dense_kernel<true><<<4 * n_sm, 256, 0, st>>>(fit, dense, grid);
    else
        em_counts_pbm_dense_kernel<false><<<grid, c.block, 0, st>>>(fit, dense, grid);
    return cudaGetLastError();
}

// Many fits in one launch: fit i owns blocks [blk_begin, blk_begin + n_blocks),
// each a contiguous chunk of kCountChunk of its qd, so a block serves one fit
// and the fit's last block runs its public M-step.  (16 bin copies here, 8 in
// the one-fit kernel: the batch's short-lived blocks gained from more copies,
// the one-fit kernel's long grid-stride blocks lost occupancy to them.)
__global__ void __launch_bounds__(256, 7) em_counts_batch_kernel(const CountFitDev* __restrict__ fits, int n_fits) {
    __shared__ int s_fit;
    if (threadIdx.x == 0) {
        int lo = 0, hi = n_fits - 1;  // last fit with blk_begin <= blockIdx.x
        while (lo < hi) {
            const int mid = (lo + hi + 1) / 2;
            if (fits[mid].blk_begin <= (int)blockIdx.x) lo = mid; else hi = mid - 1;
        }
        s_fit = lo;
    }
    __syncthreads();
    const CountFitDev cf = fits[s_fit];
    const int64_t q0 = (int64_t)((int)blockIdx.x - cf.blk_begin) * kCountChunk;
    const int64_t q1 = q0 + kCountChunk < cf.n_qd ? q0 + kCountChunk : cf.n_qd;
    count_iteration<16, 4>(*cf.fit, cf.off, cf.ent, q0 + threadIdx.x, q1, blockDim.x, (unsigned)cf.n_blocks);
}

cudaError_t launch_em_counts_batch(const CountFitDev* fits, int n_fits, int total_blocks, cudaStream_t st) {
    if (n_fits == 0 || total_blocks == 0) return cudaSuccess;
    em_counts_batch_kernel<<<total_blocks, 256, 0, st>>>(fits, n_fits);
    return cudaGetLastError();
}

}  // namespace mcd
