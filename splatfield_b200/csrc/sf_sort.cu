// Onesweep LSD radix sort and decoupled-look-back prefix scan (sm_100a).
//
// Replaces crates/sort/src/sort.rs (count_kernel + scan + scatter_plane_kernel
// per 6-bit digit, 3 launches a digit) and crates/sort/src/scan.rs
// (block_sums + scan_serial + apply_block_offsets). Design (Adinets & Merrill,
// "Onesweep: A Faster Least Significant Digit Radix Sort for GPUs", 2022):
//  * one upfront kernel reads the keys once and builds the 256-bin histogram
//    of every 8-bit digit position;
//  * one kernel per digit: a partition of 4096 keys (8192 from 2M keys on)
//    is ranked in registers and shared memory (stable warp ranking by lane
//    masks), publishes its digit counts, goes into shared memory in sorted
//    order, resolves its global digit offsets by decoupled look-back over the
//    preceding partitions, and is written out, each digit's run contiguously.
//    10M random pairs, 32 bits: 0.440 -> 0.313 ms for the whole sort (1M 89 ->
//    75 us, 1k 50 -> 44 us) against ballot ranking with the look-back before
//    the shared scatter and one shared counter per histogram bin.
// Partition indices come from an atomic ticket in launch order, so a block
// only ever waits on blocks that already hold a ticket (forward progress).
// Every wait is bounded: after kSpinLimit polls the block records
// SF_DEV_ERR_TIMEOUT in the error word and carries on, so a lost predecessor
// can corrupt the result but never hang the GPU.
#include <cstdint>
#include <type_traits>
#include <string>
#include "sf_handles.h"

namespace sfk {

namespace {

// Digit width: 4 to 8 bits (a template parameter of the kernels); the
// scratch is laid out for the widest case, 256 bins, 4 passes of 32 bits.
constexpr int kRadixBits = 8;
constexpr int kRadix = 1 << kRadixBits;
constexpr int kHistWords = 1024;  // passes x bins <= 1024 for every width
constexpr int kThreads = 256;
constexpr int kItems = 16;
constexpr int kWarps = kThreads / 32;
// Digit passes: partitions of THREADS x 16 keys. The look-back chain across
// partitions bounds a large pass (a partition publishes its inclusive prefix
// only after its own look-back), so from kWidePassN keys on the partitions
// are 8192 keys of 512 threads (half the chain);
// smaller sorts keep 4096-key partitions of 256 threads, whose single
// partitions finish sooner (1k-500k keys 12-17% faster than the wide form).
// The keys and values staged for the scatter are dynamic shared memory.
constexpr uint32_t kWidePassN = 1u << 21;
constexpr int kMinPassTile = 256 * kItems;  // look-back space is sized for it
constexpr uint32_t kFlagAgg = 1u << 30;
constexpr uint32_t kFlagPrefix = 2u << 30;
constexpr uint32_t kCountMask = (1u << 30) - 1u;
constexpr uint32_t kSpinLimit = 1u << 22;

// Test knobs of the look-back waits, set by sf_debug_lookback and passed to
// the kernels only by the standalone sort and scan entry points (the frame
// and round paths always pass zeros). spin_limit caps the polls of one wait
// (0: kSpinLimit). withhold = 1 keeps partition 0 of the scan and of every
// digit pass from publishing its status, a flag that nothing then sets: every
// later partition's wait runs out after spin_limit polls, records
// SF_DEV_ERR_TIMEOUT and returns, and the host reports SF_ERR_TIMEOUT. Every
// access stays inside the buffers either way; only the values are wrong.
LookbackKnobs g_test_knobs = {0u, 0u};

__device__ __forceinline__ uint32_t ld_relaxed(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed(uint32_t* p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned long long ld_relaxed64(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed64(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Decoupled look-back from partition `part` over one digit's status words
// stat[p * stride] (flag in the top two bits: 0 = not ready, aggregate,
// inclusive prefix), by the LPD lanes of a warp that share the digit: slot s
// (this lane's place among them) reads the kWindow predecessors after the
// kWindow * s nearest ones, so one L2 round trip covers LPD * kWindow
// partitions. All partitions of a wave publish their aggregates at about the
// same time, so a partition i places into the wave waits about
// i / (2 LPD kWindow) round trips for its prefix, and this chain is what
// bounds a large pass. Every lane of the group returns the exclusive prefix.
// A poll that finds nothing new backs off with __nanosleep (32 ns, doubling
// to 256 ns), so waiting blocks leave issue slots and L2 bandwidth to the
// partitions still ranking; a wait that outlasts kSpinLimit polls (about a
// second with the naps) records SF_DEV_ERR_TIMEOUT and returns what it has.
// Every lane of the warp must call it (the groups leave the loop together).
constexpr int kWindow = 4;
template <int LPD>
__device__ __forceinline__ uint32_t lookback_digit(const uint32_t* stat, size_t stride, uint32_t part, bool active,
                                                   uint32_t* err, uint32_t spin_limit) {
    static_assert(LPD == 1 || LPD == 2, "lanes per digit");
    const uint32_t slot = LPD == 2 ? (threadIdx.x & 31u) >> 4 : 0u;
    uint32_t excl = 0, spins = 0, nap = 32;
    const uint32_t limit = spin_limit ? spin_limit : kSpinLimit;
    int32_t p = active ? (int32_t)part - 1 : -1;
    while (__any_sync(0xffffffffu, p >= 0)) {
        uint32_t st[kWindow];
        const int32_t q = p - (int32_t)slot * kWindow;
#pragma unroll
        for (int w = 0; w < kWindow; ++w)
            st[w] = (p >= 0 && q - w >= 0) ? ld_relaxed(stat + (size_t)(q - w) * stride) : kFlagPrefix;
        uint32_t sum = 0, used = 0;
        bool open = true, found = false;
#pragma unroll
        for (int w = 0; w < kWindow; ++w) {
            open = open && (st[w] & ~kCountMask) != 0;
            if (open) {
                sum += st[w] & kCountMask;
                ++used;
                found = (st[w] & ~kCountMask) == kFlagPrefix;
                open = !found;
            }
        }
        if (LPD == 2) {
            const uint32_t osum = __shfl_xor_sync(0xffffffffu, sum, 16);
            const uint32_t oused = __shfl_xor_sync(0xffffffffu, used, 16);
            const bool ofound = __shfl_xor_sync(0xffffffffu, (uint32_t)found, 16) != 0;
            const uint32_t s0 = slot ? osum : sum, s1 = slot ? sum : osum;
            const uint32_t u0 = slot ? oused : used, u1 = slot ? used : oused;
            const bool f0 = slot ? ofound : found, f1 = slot ? found : ofound;
            const bool both = !f0 && u0 == kWindow;
            sum = s0 + (both ? s1 : 0u);
            used = u0 + (both ? u1 : 0u);
            found = f0 || (both && f1);
        }
        if (p >= 0) {
            excl += sum;
            p -= (int32_t)used;
            if (found) p = -1;
        }
        if (p >= 0 && used == 0) {
            if (++spins > limit) {
                atomicOr(err, SF_DEV_ERR_TIMEOUT);
                p = -1;
            } else {
                __nanosleep(nap);
                nap = min(nap * 2u, 256u);
            }
        }
    }
    return excl;
}

__device__ __forceinline__ uint32_t lanemask_lt() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

__device__ __forceinline__ uint32_t load_n(const uint32_t* n_dev, uint32_t n_static) {
    return n_dev ? *n_dev : n_static;
}

// Upfront digit histograms: hist[pass * 2^BITS + digit] over all n keys.
template <int BITS>
__global__ __launch_bounds__(kThreads) void radix_histogram_kernel(
    const uint32_t* __restrict__ keys, const uint32_t* n_dev, uint32_t n_static,
    uint32_t num_passes, uint32_t bits, uint32_t* __restrict__ hist) {
    constexpr uint32_t R = 1u << BITS;
    __shared__ uint32_t s_hist[kHistWords];
    const uint32_t n = load_n(n_dev, n_static);
    for (uint32_t i = threadIdx.x; i < num_passes * R; i += kThreads) s_hist[i] = 0;
    __syncthreads();
    // Whole warps iterate together (the bound is rounded up) so that runs of
    // equal digits in neighbouring lanes are merged before the shared atomic:
    // emitted tile ids come in runs, and 32 lanes on one bin would otherwise
    // serialise. A lane whose digit differs from its left neighbour's adds the
    // length of its run.
    // Each warp takes 128 consecutive keys per step (4 loads in flight per
    // lane, each covering 32 consecutive keys across the lanes).
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t warp_global = (blockIdx.x * kThreads + threadIdx.x) >> 5;
    const uint32_t warps_total = (gridDim.x * kThreads) >> 5;
    for (uint32_t base = warp_global * 128u; base < n; base += warps_total * 128u) {
        uint32_t kk[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint32_t i = base + u * 32u + lane;
            kk[u] = i < n ? keys[i] : 0u;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const bool valid = base + u * 32u + lane < n;
            for (uint32_t p = 0; p < num_passes; ++p) {
                const uint32_t shift = p * BITS;
                const uint32_t w = bits - shift < (uint32_t)BITS ? bits - shift : (uint32_t)BITS;
                const uint32_t d = valid ? ((kk[u] >> shift) & ((1u << w) - 1u)) : R;
                const uint32_t left = __shfl_up_sync(0xffffffffu, d, 1);
                const bool head = lane == 0 || left != d;
                const uint32_t heads = __ballot_sync(0xffffffffu, head);
                if (valid && head) {
                    const uint32_t above = heads & ~((2u << lane) - 1u);
                    const uint32_t next = above ? (uint32_t)(__ffs(above) - 1) : 32u;
                    atomicAdd(&s_hist[p * R + d], next - lane);
                }
            }
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < num_passes * R; i += kThreads)
        if (s_hist[i]) atomicAdd(&hist[i], s_hist[i]);
}

// The same counts from kWideHistN keys on. A shared atomic costs a cycle per
// lane on the busiest bank, so with one counter per bin the random digits of a
// warp serialise about four deep and four digits per key took 62 us for 10M
// keys. Here lane l counts in column l of a 32-column table (bank l whatever
// the digit, equal digits of a warp included): 24 us. The table
// (up to 128 KB) allows one CTA of 1024 threads per SM, and clearing and
// summing it costs about 3 us, so smaller inputs keep the form above.
constexpr uint32_t kWideHistN = 1u << 20;
constexpr int kWideHistThreads = 1024;
template <int BITS>
__global__ __launch_bounds__(kWideHistThreads, 1) void radix_histogram_wide_kernel(
    const uint32_t* __restrict__ keys, const uint32_t* n_dev, uint32_t n_static, uint32_t num_passes, uint32_t bits,
    uint32_t* __restrict__ hist) {
    constexpr uint32_t R = 1u << BITS;
    constexpr int kLoads = 8;
    extern __shared__ __align__(16) uint32_t s_cols[];
    const uint32_t n = load_n(n_dev, n_static);
    const uint32_t bins = num_passes * R, tid = threadIdx.x, lane = tid & 31u;
    for (uint32_t i = tid; i < bins * 8; i += kWideHistThreads)
        reinterpret_cast<uint4*>(s_cols)[i] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    const uint32_t last_mask = (1u << (bits - (num_passes - 1) * BITS)) - 1u;
    const uint32_t warps = (gridDim.x * kWideHistThreads) >> 5;
    for (uint64_t base = (uint64_t)((blockIdx.x * kWideHistThreads + tid) >> 5) * (32 * kLoads); base < n;
         base += (uint64_t)warps * (32 * kLoads)) {
        uint32_t kk[kLoads];
#pragma unroll
        for (int u = 0; u < kLoads; ++u) {
            const uint64_t i = base + u * 32 + lane;
            kk[u] = i < n ? __ldg(keys + i) : 0u;
        }
#pragma unroll
        for (int u = 0; u < kLoads; ++u) {
            if (base + u * 32 + lane >= n) continue;
            for (uint32_t p = 0; p < num_passes; ++p) {
                const uint32_t d = (kk[u] >> (p * BITS)) & (p + 1 < num_passes ? R - 1u : last_mask);
                atomicAdd(&s_cols[(p * R + d) * 32 + lane], 1u);
            }
        }
    }
    __syncthreads();
    for (uint32_t i = tid; i < bins; i += kWideHistThreads) {
        uint32_t sum = 0;
#pragma unroll
        for (uint32_t c = 0; c < 32; ++c) sum += s_cols[i * 32 + ((c + lane) & 31u)];
        if (sum) atomicAdd(&hist[i], sum);
    }
}

// Shared memory of one digit pass.
template <int BITS, int THREADS>
struct PassShared {
    static constexpr uint32_t R = 1u << BITS;
    uint32_t keys[THREADS * kItems], vals[THREADS * kItems];  // staged for the scatter
    // Per warp and digit: the lanes of the item being ranked that hold the
    // digit; the warp's keys of it so far, later the first staged slot of the
    // warp's keys of it.
    uint32_t lanes[THREADS / 32][R], warp[THREADS / 32][R];
    uint32_t base[R], gstart[R], total[R];
    uint32_t scan[THREADS / 32];
    uint32_t part;
};

// Exclusive prefix of v over the block's threads (two barriers; s_scan is
// free again after the caller's next barrier).
template <int THREADS>
__device__ __forceinline__ uint32_t block_exclusive(uint32_t v, uint32_t* s_scan) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += t;
    }
    __syncthreads();
    if (lane == 31) s_scan[warp] = incl;
    __syncthreads();
    const uint32_t before = lane < warp ? s_scan[lane] : 0u;  // warp < 32
    return incl - v + __reduce_add_sync(0xffffffffu, before);
}

// One partition of a digit pass; FULL: all THREADS x kItems keys exist.
template <int BITS, int THREADS, bool FULL>
__device__ __forceinline__ void onesweep_partition(
    PassShared<BITS, THREADS>& sm, const uint32_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
    uint32_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out, uint32_t n, uint32_t part, uint32_t shift,
    uint32_t digit_mask, const uint32_t* __restrict__ pass_hist, uint32_t* lookback, uint32_t* err, int vals_iota,
    int write_keys, LookbackKnobs knobs) {
    constexpr uint32_t R = 1u << BITS;
    constexpr int kPassWarps = THREADS / 32, kPassTile = THREADS * kItems;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t base = part * kPassTile;
    const uint32_t w0 = base + warp * (kItems * 32) + lane;  // this lane's item i is w0 + 32 i

    uint32_t k[kItems];
#pragma unroll
    for (int i = 0; i < kItems; ++i) k[i] = FULL || w0 + i * 32 < n ? keys_in[w0 + i * 32] : 0u;
    // Stable warp ranking, items in index order, lanes in lane order: each
    // lane sets its bit in its digit's lane mask; the mask gives its rank
    // among the item's equal digits, and the first lane of a digit adds them
    // to the warp's count and clears the mask. Against one ballot per digit
    // bit (8 votes and 24 more instructions an item), which left the pass
    // bound by issue slots, this one is bound by shared-memory bank conflicts
    // (LSU pipe 69% busy, issue 35%): a pass over 10M pairs 84 -> 70 us. With
    // 6, 10 or all 16 of a thread's items ranked by ballots instead, the
    // 10M-key sort took 0.315, 0.336 and 0.361 ms against 0.313. rank < 512 (a
    // warp's keys): two to a word.
    const uint32_t lt = lanemask_lt(), me = 1u << lane;
    uint32_t rank[kItems / 2];
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
        const bool valid = FULL || w0 + i * 32 < n;
        const uint32_t d = (k[i] >> shift) & digit_mask;
        uint32_t *count = &sm.warp[warp][d], *lanes = &sm.lanes[warp][d];
        if (valid) atomicOr(lanes, me);
        __syncwarp();
        const uint32_t m = *lanes, before = *count;
        __syncwarp();
        if (valid && (m & lt) == 0) {
            *lanes = 0u;
            *count = before + (uint32_t)__popc(m);
        }
        const uint32_t r = before + (uint32_t)__popc(m & lt);
        rank[i / 2] = i % 2 == 0 ? r : rank[i / 2] | (r << 16);
        __syncwarp();
    }
    __syncthreads();

    // Per digit: the block's count, published; the first staged slot of each
    // warp's keys of it; the digit's first global slot.
    uint32_t digit_total = 0;
    if (tid < R) {
#pragma unroll
        for (int w = 0; w < kPassWarps; ++w) digit_total += sm.warp[w][tid];
        if (part > 0 || !knobs.withhold)
            st_relaxed(&lookback[(size_t)part * R + tid], (part == 0 ? kFlagPrefix : kFlagAgg) | digit_total);
    }
    const uint32_t local = block_exclusive<THREADS>(digit_total, sm.scan);
    const uint32_t global = block_exclusive<THREADS>(tid < R ? pass_hist[tid] : 0u, sm.scan);
    if (tid < R) {
        uint32_t run = local;
#pragma unroll
        for (int w = 0; w < kPassWarps; ++w) {
            const uint32_t c = sm.warp[w][tid];
            sm.warp[w][tid] = run;
            run += c;
        }
        sm.total[tid] = digit_total;
        sm.gstart[tid] = global - local;
    }
    __syncthreads();
    // Into shared memory in the partition's sorted order, which needs no
    // global offset: keys, then values, leave their registers before the
    // look-back (with both held through it the compiler spilled 36 words).
    // The digits are formed anew (the empty asm hides that they were known):
    // sixteen kept slot addresses would be spilled.
    uint32_t shift2 = shift;
    asm volatile("" : "+r"(shift2));
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
        if (FULL || w0 + i * 32 < n) {
            const uint32_t pos = sm.warp[warp][(k[i] >> shift2) & digit_mask] + ((rank[i / 2] >> (i % 2 * 16)) & 0xffffu);
            sm.keys[pos] = k[i];
            k[i] = pos;
        }
    }
    uint32_t v[kItems];
#pragma unroll
    for (int i = 0; i < kItems; ++i)
        v[i] = vals_iota ? w0 + i * 32 : (FULL || w0 + i * 32 < n ? vals_in[w0 + i * 32] : 0u);
#pragma unroll
    for (int i = 0; i < kItems; ++i)
        if (FULL || w0 + i * 32 < n) sm.vals[k[i]] = v[i];
    {
        constexpr int LPD = THREADS >= 2 * (int)R ? 2 : 1;
        const uint32_t d = LPD == 2 ? warp * 16 + (lane & 15u) : tid;
        const bool active = d < R;
        uint32_t* stat = lookback + (active ? d : 0u);
        const uint32_t excl = lookback_digit<LPD>(stat, R, part, active, err, knobs.spin_limit);
        if (active && (LPD == 1 || lane < 16)) {
            if (part > 0) st_relaxed(&stat[(size_t)part * R], kFlagPrefix | ((excl + sm.total[d]) & kCountMask));
            sm.base[d] = sm.gstart[d] + excl;
        }
    }
    __syncthreads();
    const uint32_t cnt = FULL ? (uint32_t)kPassTile : n - base;
#pragma unroll 4
    for (uint32_t j = tid; j < cnt; j += THREADS) {
        const uint32_t key = sm.keys[j];
        const uint32_t out = sm.base[(key >> shift) & digit_mask] + j;
        if (out >= n) continue;  // only after a timed-out look-back
        if (write_keys) keys_out[out] = key;
        vals_out[out] = sm.vals[j];
    }
}

// One BITS-bit digit pass. `vals_iota` substitutes vals_in[i] = i.
template <int BITS, int THREADS>
__global__ __launch_bounds__(THREADS, THREADS >= 512 ? 2 : 4) void onesweep_pass_kernel(
    const uint32_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
    uint32_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out, const uint32_t* n_dev,
    uint32_t n_static, uint32_t shift, uint32_t digit_mask, const uint32_t* __restrict__ pass_hist,
    uint32_t* lookback, uint32_t* ticket, uint32_t* err, int vals_iota, int write_keys, LookbackKnobs knobs) {
    constexpr uint32_t R = 1u << BITS;
    constexpr int kPassTile = THREADS * kItems;
    static_assert(THREADS >= (int)R, "one thread per digit");
    extern __shared__ __align__(16) unsigned char s_pass[];
    PassShared<BITS, THREADS>& sm = *reinterpret_cast<PassShared<BITS, THREADS>*>(s_pass);
    const uint32_t tid = threadIdx.x;
    const uint32_t n = load_n(n_dev, n_static);
    const uint32_t num_parts = (n + kPassTile - 1) / kPassTile;
    if (tid == 0) sm.part = atomicAdd(ticket, 1u);
    for (uint32_t i = tid; i < THREADS / 32 * R; i += THREADS) (&sm.warp[0][0])[i] = (&sm.lanes[0][0])[i] = 0u;
    __syncthreads();
    const uint32_t part = sm.part;
    if (part >= num_parts) return;
    if (n - part * kPassTile >= (uint32_t)kPassTile)
        onesweep_partition<BITS, THREADS, true>(sm, keys_in, vals_in, keys_out, vals_out, n, part, shift, digit_mask,
                                                pass_hist, lookback, err, vals_iota, write_keys, knobs);
    else
        onesweep_partition<BITS, THREADS, false>(sm, keys_in, vals_in, keys_out, vals_out, n, part, shift,
                                                 digit_mask, pass_hist, lookback, err, vals_iota, write_keys, knobs);
}

// The scan's look-back done by one whole warp: lane l reads the status of
// partition p - l (p the newest predecessor not yet summed), so one L2 round
// trip covers 32 predecessors. If some lane finds an inclusive prefix and
// every lane before it an aggregate, the warp sums those lanes and stops;
// otherwise it sums the aggregates before the first lane whose partition
// has published nothing and reads again from there, with the same backoff
// and bound as lookback_digit. Lanes past partition 0 read a zero prefix.
// Returns the exclusive prefix in every lane.
__device__ unsigned long long lookback_warp64(const unsigned long long* stat, uint32_t part, uint32_t* err,
                                              uint32_t spin_limit, unsigned long long flag_prefix,
                                              unsigned long long value_mask) {
    const uint32_t lane = threadIdx.x & 31u;
    unsigned long long excl = 0;
    int64_t p = (int64_t)part - 1;
    uint32_t spins = 0, nap = 32;
    const uint32_t limit = spin_limit ? spin_limit : kSpinLimit;
    while (p >= 0) {
        const int64_t q = p - (int64_t)lane;
        const unsigned long long st = q >= 0 ? ld_relaxed64(stat + q) : flag_prefix;
        const unsigned long long flag = st & ~value_mask;
        const uint32_t not_ready = __ballot_sync(0xffffffffu, flag == 0);
        const uint32_t prefix = __ballot_sync(0xffffffffu, flag == flag_prefix);
        const uint32_t first_nr = not_ready ? (uint32_t)(__ffs(not_ready) - 1) : 32u;
        const uint32_t first_pf = prefix ? (uint32_t)(__ffs(prefix) - 1) : 32u;
        const bool done = first_pf < first_nr;
        const uint32_t take = done ? first_pf + 1 : first_nr;
        unsigned long long v = lane < take ? (st & value_mask) : 0ull;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        excl += v;
        if (done) break;
        if (take == 0) {
            if (++spins > limit) {
                if (lane == 0) atomicOr(err, SF_DEV_ERR_TIMEOUT);
                break;
            }
            __nanosleep(nap);
            nap = min(nap * 2u, 256u);
        }
        p -= take;
    }
    return excl;
}

// Single-pass exclusive scan with optional gather:
// out[i] = sum_{j<i} counts[gids ? gids[j] : j], 64-bit running sums, the
// u32 low word stored; *total_out = the 64-bit total.
constexpr int kScanItems = 16;
constexpr int kScanTile = kThreads * kScanItems;
constexpr unsigned long long kScanFlagAgg = 1ull << 62;
constexpr unsigned long long kScanFlagPrefix = 2ull << 62;
constexpr unsigned long long kScanValMask = (1ull << 62) - 1ull;

__global__ __launch_bounds__(kThreads) void scan_kernel(
    const uint32_t* __restrict__ gids, const uint32_t* counts, uint32_t* out, const uint32_t* n_dev,
    uint32_t n_static, unsigned long long* lookback, uint32_t* ticket,
    unsigned long long* total_out, uint32_t* err, LookbackKnobs knobs) {
    pdl_trigger();
    pdl_wait();
    __shared__ uint32_t s_part;
    __shared__ unsigned long long s_warp[kWarps];
    __shared__ unsigned long long s_prefix;
    __shared__ uint32_t s_tile[kThreads * (kScanItems + 1)];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t n = load_n(n_dev, n_static);
    const uint32_t num_parts = (n + kScanTile - 1) / kScanTile;
    if (tid == 0) s_part = atomicAdd(ticket, 1u);
    __syncthreads();
    const uint32_t part = s_part;
    if (n == 0) {
        if (part == 0 && tid == 0 && total_out) *total_out = 0ull;
        return;
    }
    if (part >= num_parts) return;
    // Coalesced striped loads, transposed through shared memory so each
    // thread scans kScanItems consecutive elements (row pitch 17 words keeps
    // the transposed reads conflict-free).
    const uint32_t tile0 = part * kScanTile;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        const uint32_t e = i * kThreads + tid;
        const uint32_t idx = tile0 + e;
        uint32_t c = 0;
        if (idx < n) c = counts[gids ? gids[idx] : idx];
        s_tile[(e / kScanItems) * (kScanItems + 1) + e % kScanItems] = c;
    }
    __syncthreads();
    const uint32_t base = tile0 + tid * kScanItems;
    uint32_t v[kScanItems];
    unsigned long long local = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        v[i] = s_tile[tid * (kScanItems + 1) + i];
        local += v[i];
    }
    // Block exclusive scan of the per-thread sums.
    unsigned long long incl = local;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += t;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    unsigned long long warp_prefix = 0, block_total = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
        if ((uint32_t)w < warp) warp_prefix += s_warp[w];
        block_total += s_warp[w];
    }
    if (warp == 0) {
        unsigned long long excl = 0;
        if (part == 0) {
            if (lane == 0 && !knobs.withhold) st_relaxed64(&lookback[0], kScanFlagPrefix | block_total);
        } else {
            if (lane == 0) st_relaxed64(&lookback[part], kScanFlagAgg | block_total);
            excl = lookback_warp64(lookback, part, err, knobs.spin_limit, kScanFlagPrefix, kScanValMask);
            if (lane == 0) st_relaxed64(&lookback[part], kScanFlagPrefix | (excl + block_total));
        }
        if (lane == 0) {
            s_prefix = excl;
            if (part == num_parts - 1 && total_out) *total_out = excl + block_total;
        }
    }
    __syncthreads();
    unsigned long long running = s_prefix + warp_prefix + (incl - local);
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        s_tile[tid * (kScanItems + 1) + i] = (uint32_t)running;
        running += v[i];
    }
    (void)base;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        const uint32_t e = i * kThreads + tid;
        const uint32_t idx = tile0 + e;
        if (idx < n) out[idx] = s_tile[(e / kScanItems) * (kScanItems + 1) + e % kScanItems];
    }
}

}  // namespace

uint32_t radix_passes(uint32_t bits, uint32_t digit_bits) { return (bits + digit_bits - 1) / digit_bits; }

size_t radix_temp_bytes(uint32_t max_elems, uint32_t max_passes) {
    const size_t parts = (max_elems + kMinPassTile - 1) / kMinPassTile;
    // hist [1024] + tickets [16] + lookback [passes][parts][256]: 32-bit keys
    // at 8-bit digits (4 passes x 256 bins) need the most, and every narrower
    // digit (passes x bins <= 1024) fits the same space.
    return kHistWords * 4 + 64 + (size_t)max_passes * parts * kRadix * 4;
}

namespace {

template <int BITS>
cudaError_t radix_sort_bits(const uint32_t* keys_in, const uint32_t* vals_in, uint32_t* keys_a, uint32_t* vals_a,
                            uint32_t* keys_b, uint32_t* vals_b, uint32_t n, const uint32_t* n_dev, uint32_t max_n,
                            uint32_t bits, bool write_keys, bool vals_iota, void* temp, uint32_t* err,
                            int sm_count, cudaStream_t stream, int* out_in_b, LookbackKnobs knobs) {
    constexpr uint32_t R = 1u << BITS;
    const uint32_t passes = radix_passes(bits, BITS);
    const uint32_t grid_n = n_dev ? max_n : n;
    uint8_t* t = static_cast<uint8_t*>(temp);
    uint32_t* hist = reinterpret_cast<uint32_t*>(t);
    uint32_t* tickets = reinterpret_cast<uint32_t*>(t + kHistWords * 4);
    uint32_t* lookback = reinterpret_cast<uint32_t*>(t + kHistWords * 4 + 64);
    const bool wide = grid_n >= kWidePassN;
    const uint32_t tile = (wide ? 512u : 256u) * kItems;
    const size_t parts = (grid_n + tile - 1) / tile;
    cudaError_t e = cudaMemsetAsync(temp, 0, kHistWords * 4 + 64 + passes * parts * R * 4, stream);
    if (e != cudaSuccess) return e;
    if (parts == 0) { *out_in_b = 0; return cudaSuccess; }
    if (grid_n >= kWideHistN) {
        // The limit is one per kernel and device: always set for the most
        // passes, so that no call lowers it under another thread's launch.
        const size_t smem = (size_t)passes * R * 32 * 4;
        e = cudaFuncSetAttribute(radix_histogram_wide_kernel<BITS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 kHistWords * 32 * 4);
        if (e != cudaSuccess) return e;
        radix_histogram_wide_kernel<BITS><<<(uint32_t)std::max(sm_count, 1), kWideHistThreads, smem, stream>>>(
            keys_in, n_dev, n, passes, bits, hist);
    } else {
        const uint32_t hist_blocks = (uint32_t)std::min<size_t>((grid_n + kThreads * 8 - 1) / (kThreads * 8),
                                                                 (size_t)sm_count * 4);
        radix_histogram_kernel<BITS><<<std::max(hist_blocks, 1u), kThreads, 0, stream>>>(
            keys_in, n_dev, n, passes, bits, hist);
    }
    int in_b = 0;
    auto run_passes = [&](auto threads) -> cudaError_t {
        constexpr int TH = decltype(threads)::value;
        cudaError_t e2 = cudaFuncSetAttribute(onesweep_pass_kernel<BITS, TH>,
                                              cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(PassShared<BITS, TH>));
        if (e2 != cudaSuccess) return e2;
        const uint32_t* kin = keys_in;
        const uint32_t* vin = vals_in;
        for (uint32_t p = 0; p < passes; ++p) {
            const uint32_t shift = p * BITS;
            const uint32_t w = std::min<uint32_t>(bits - shift, BITS);
            uint32_t* kout = (p % 2 == 0) ? keys_a : keys_b;
            uint32_t* vout = (p % 2 == 0) ? vals_a : vals_b;
            const bool wk = write_keys || (p + 1 < passes);
            onesweep_pass_kernel<BITS, TH><<<(uint32_t)parts, TH, sizeof(PassShared<BITS, TH>), stream>>>(
                kin, vin, kout, vout, n_dev, n, shift, (1u << w) - 1u, hist + p * R,
                lookback + (size_t)p * parts * R, tickets + p, err, (vals_iota && p == 0) ? 1 : 0,
                wk ? 1 : 0, knobs);
            kin = kout;
            vin = vout;
            in_b = (p % 2 == 1);
        }
        return cudaSuccess;
    };
    e = wide ? run_passes(std::integral_constant<int, 512>{}) : run_passes(std::integral_constant<int, 256>{});
    if (e != cudaSuccess) return e;
    *out_in_b = in_b;
    note_launches(1 + passes);
    return cudaGetLastError();
}

}  // namespace

cudaError_t radix_sort_pairs(const uint32_t* keys_in, const uint32_t* vals_in, uint32_t* keys_a,
                             uint32_t* vals_a, uint32_t* keys_b, uint32_t* vals_b, uint32_t n,
                             const uint32_t* n_dev, uint32_t max_n, uint32_t bits, bool write_keys,
                             bool vals_iota, void* temp, uint32_t* err, int sm_count,
                             cudaStream_t stream, int* out_in_b, LookbackKnobs knobs, uint32_t digit_bits) {
    switch (digit_bits) {
#define SF_RADIX_CASE(B)                                                                                      \
    case B:                                                                                                   \
        return radix_sort_bits<B>(keys_in, vals_in, keys_a, vals_a, keys_b, vals_b, n, n_dev, max_n, bits,   \
                                  write_keys, vals_iota, temp, err, sm_count, stream, out_in_b, knobs);
        SF_RADIX_CASE(4)
        SF_RADIX_CASE(5)
        SF_RADIX_CASE(6)
        SF_RADIX_CASE(7)
        SF_RADIX_CASE(8)
#undef SF_RADIX_CASE
        default: return cudaErrorInvalidValue;
    }
}

size_t scan_temp_bytes(uint32_t max_elems) {
    const size_t parts = (max_elems + kScanTile - 1) / kScanTile;
    return 64 + std::max<size_t>(parts, 1) * 8;
}

cudaError_t exclusive_scan(const uint32_t* gids, const uint32_t* counts, uint32_t* out, uint32_t n,
                           const uint32_t* n_dev, uint32_t max_n, void* temp,
                           unsigned long long* total_out, uint32_t* err, cudaStream_t stream,
                           LookbackKnobs knobs) {
    const uint32_t grid_n = n_dev ? max_n : n;
    const size_t parts = std::max<size_t>((grid_n + kScanTile - 1) / kScanTile, 1);
    uint8_t* t = static_cast<uint8_t*>(temp);
    uint32_t* ticket = reinterpret_cast<uint32_t*>(t);
    unsigned long long* lookback = reinterpret_cast<unsigned long long*>(t + 64);
    cudaError_t e = cudaMemsetAsync(temp, 0, 64 + parts * 8, stream);
    if (e != cudaSuccess) return e;
    scan_kernel<<<(uint32_t)parts, kThreads, 0, stream>>>(gids, counts, out, n_dev, n, lookback,
                                                           ticket, total_out, err, knobs);
    note_launches(1);
    return cudaGetLastError();
}

}  // namespace sfk

namespace sfk {
LookbackKnobs lookback_test_knobs() { return g_test_knobs; }
}  // namespace sfk

extern "C" int sf_debug_lookback(uint32_t spin_limit, int withhold) {
    sfk::g_test_knobs = sfk::LookbackKnobs{spin_limit, withhold ? 1u : 0u};
    return SF_OK;
}

extern "C" int sf_debug_giant_lists(uint32_t lists) {
    sfk::set_giant_max_lists(lists);
    return SF_OK;
}
