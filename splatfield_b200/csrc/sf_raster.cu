// Tile rasterizer for sm_100a: rasterize_kernel (src/raster.rs:88-230) in its
// RGB, total-responsibility and evidence modes, plus mode 3, the adjoint of a
// per-splat scalar feature.
//
// A CTA owns all (CTAS = 1) or part (CTAS = 2, 4) of one 16x16 tile: warp w of
// the tile covers the 8x4 pixel block at ((w & 1) * 8, (w >> 1) * 4), and a
// CTA of 256 / CTAS threads takes 8 / CTAS consecutive warps of it. Every
// CTA walks the tile's whole list in order for its own pixels, so splitting a
// tile changes no pixel's walk and no result; a long, unsaturated list is
// then walked by several SMs at once.
//
// Staging: the splat records of the list are gathered 256 entries at a time
// into shared memory with cp.async (16-byte global -> shared copies that
// need no registers), double-buffered: chunk c + 1 is in flight while chunk c
// is composited, and the ids of chunk c + 2 are loaded a chunk ahead, so the
// gather latency overlaps the walk. One barrier per chunk, with the saturation
// count: past it chunk c is complete and chunk c - 1's buffer is free (mode 3
// takes a second one, for its single-buffered sums).
//
// Per pair: the power of the splat's quadratic form at the pixel; a pair with
// power above the splat's power_max (alpha < 1/255 for sure) is skipped;
// alpha = min(opacity * exp(-power), 0.999), pairs below 1/255 are skipped,
// and the pixel stops after the contributor that takes T below 1/255
// (src/raster.rs:173-221). The f32 operations are the oracle's, in the same
// order (sf_math.cuh), so images and words are bit-identical to it.
//
// What bounds the walk is instruction issue (about 65% of the slots at 1080p,
// the rest barriers and the tail of long tiles), so it takes two entries at a
// time: a warp packs the entries it walks into pair records (PairRec), and the
// two powers and exponentials are one chain of packed f32 operations, which
// round each half as the scalar ones do. Only the composite itself stays in
// list order, and it is written with predicates. 1M splats at 1080p: 178 ->
// 160 us and 127M -> 108M warp instructions against packed pairs with branches
// in the composite, and 190 us with one entry at a time; 3001 splats at 97x61,
// where the chain's latency counts, 43 -> 27 us. A limit of 48 registers (five
// CTAs an SM instead of four) spilled 12 words and took 173 us.
//
// CULL: each warp walks only the entries that can reach its 8x4 block (the
// power_max box from the projection, then the exact test of sf_tile.cuh), 32
// candidates per ballot; a skipped pair has power above power_max, which the
// per-pixel test skips anyway, so nothing changes but the work. Every frame
// takes this form: most entries of a tile's list miss most of its eight blocks
// (against walking every entry: 3001 splats at 97x61, 73 -> 43 us; 50k splats
// at 333x217 with the adjoint's state, 68 -> 43 us). The walk over every entry remains for the pair
// diagnostics (detail), which count what each form visits.
//
// Responsibility / evidence words: the 32 pixels' fixed-point shares of an
// entry are summed by the warp (redux.sync) only when one of them is non-zero,
// added to a per-entry shared accumulator, and the chunk's accumulators go to
// global memory with one atomic per splat per CTA. Integer sums are
// order-independent, so the words equal the reference's per-pixel atomics.
//
// Mode 3: for the render F(p) = sum_k f_k alpha_k T_k of a per-splat scalar
// feature f, dF(p)/df_k = alpha_k T_k, so for L = sum_p w(p) F(p) the gradient
// dL/df_i = sum_p w(p) alpha_i T_i(p): splat i's responsibility weighted by w.
// Both factors are at hand in the forward walk, so one pass gives the two
// sums w_fg = mask(p) and w_bg = 1 - mask(p) (no mask: all in fg), the
// real-valued form of the words that modes 1 and 2 truncate per pixel, and
// T comes from the forward product alone. Up to four walked entries are summed
// over the warp together (warp_sum_scatter: 6 shuffles for 4 sums, 9 for 8,
// where a block straddles the mask's edge), each warp stores its sums in its
// own shared slots (shared f32 atomics are compare-and-swap loops), and the
// flush adds the eight warps' slots and goes to global memory with one atomic
// per splat, weight and CTA. The order of those atomics is not fixed.
// A transmittance-only pass and a back-to-front replay of every entry, as two
// kernels, took 400 + 1300 us for a 384x384 view of 3M splats; in one pass the
// 16-view round of such views went from 12.1 to 8.7 ms.
//
// LAZY: the tile's list comes unsorted (the binned build's placed (depth key,
// splat id) pairs) and is put in order here, slab by slab, only as far as the
// pixels need: a 256-bin histogram over the 64-bit (key, id) values left
// picks a run of bins holding at most kSlab entries, that slab is gathered and
// bitonic-sorted in shared memory and composited, and the next slab starts
// after the last bin taken. (key, id) values are distinct and slabs end on bin
// boundaries, so the composite order is exactly the sorted list's.
#include <cstdint>
#include "sf_internal.h"
#include "sf_math.cuh"
#include "sf_tile.cuh"

namespace sfk {

namespace {

using namespace sfm;
using namespace sft;

constexpr uint32_t kChunk = 256;
constexpr uint32_t kSlab = 2048;
constexpr uint32_t kFirstSlab = 256;

// Modes: 0 RGB, 1 total responsibility words, 2 evidence (fg / bg) words,
// 3 real-valued fg / bg responsibilities.
template <int MODE>
struct ModeOf {
    static constexpr bool kColor = MODE == 0;
    static constexpr bool kWords = MODE == 1 || MODE == 2;
    static constexpr bool kReal = MODE == 3;
};

// Shared staging of one CTA: two buffers of kChunk records each.
template <int MODE, bool CULL, uint32_t NT>
struct Stage {
    static constexpr bool kC = ModeOf<MODE>::kColor, kW = ModeOf<MODE>::kWords, kR = ModeOf<MODE>::kReal;
    float4 g0[2][kChunk];
    float4 g1[2][kChunk];
    float4 col[kC ? 2 : 1][kC ? kChunk : 1];
    float2 ext[CULL ? 2 : 1][CULL ? kChunk : 1];
    uint32_t gid[kW || kR ? 2 : 1][kW || kR ? kChunk : 1];
    uint32_t acc0[kW ? 2 : 1][kW ? kChunk : 1];
    uint32_t acc1[MODE == 2 ? 2 : 1][MODE == 2 ? kChunk : 1];
    // The entries a warp walks next, two by two (PairRec).
    PairRec<kC> pairs[NT / 32][16];
    // Each warp's sums of the chunk being walked (zero when it is staged).
    float part[kR ? 2 : 1][kR ? NT / 32 : 1][kR ? kChunk : 1];
};

struct PixelState {
    float T, pr, pg, pb;
    uint32_t last;
    uint32_t n_eval, n_hit, n_proc;
};

// Composites list entries [0, count) in order for this CTA's pixels; id(i)
// gives entry i's splat id, list_off the entry's position in the tile's
// whole sorted list. (wxf, wyf): the first pixel centre of this warp's 8x4
// block. Returns true once every pixel of the CTA is saturated (uniform).
// EXACT: ps.last is the pixel's last contributor (1-based position); otherwise
// the end of the chunk it lies in, which is all that the pair statistics need
// of a list that is walked from its start.
template <int MODE, bool CULL, bool DETAIL, bool EXACT, uint32_t NT, typename IdOf>
__device__ bool composite_list(const RasterArgs& a, Stage<MODE, CULL, NT>& sm, IdOf id, uint32_t count,
                               uint32_t list_off, float fx, float fy, float wxf, float wyf, uint32_t inside,
                               PixelState& ps) {
    constexpr uint32_t kPer = kChunk / NT;
    constexpr bool kColor = ModeOf<MODE>::kColor, kWords = ModeOf<MODE>::kWords, kReal = ModeOf<MODE>::kReal;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const float inv255 = 1.0f / 255.0f;
    const uint32_t nchunks = (count + kChunk - 1) / kChunk;
    if (nchunks == 0) return false;
    uint32_t g_next[kPer];
    auto load_ids = [&](uint32_t c) {
#pragma unroll
        for (uint32_t k = 0; k < kPer; ++k) {
            const uint32_t idx = c * kChunk + k * NT + tid;
            g_next[k] = idx < count ? id(idx) : 0u;
        }
    };
    auto issue = [&](uint32_t c, uint32_t b) {
#pragma unroll
        for (uint32_t k = 0; k < kPer; ++k) {
            const uint32_t e = k * NT + tid;
            if (c * kChunk + e < count) {
                const uint32_t g = g_next[k];
                cp_async16(&sm.g0[b][e], a.geo0 + g);
                cp_async16(&sm.g1[b][e], a.geo1 + g);
                if (kColor) cp_async16(&sm.col[b][e], a.color + g);
                if (CULL) cp_async8(&sm.ext[b][e], a.ext + g);
                if (kWords || kReal) sm.gid[b][e] = g;
            }
        }
    };
    // Sums of buffer b's first cnt entries to global memory; the
    // accumulators are left at zero for the buffer's next chunk.
    auto flush = [&](uint32_t b, uint32_t cnt) {
#pragma unroll
        for (uint32_t k = 0; k < kPer; ++k) {
            const uint32_t e = k * NT + tid;
            if (kReal && e < cnt) {
                float f[2] = {0.0f, 0.0f};
#pragma unroll
                for (uint32_t x = 0; x < 2; ++x)
#pragma unroll
                    for (uint32_t w = 0; w < NT / 32; ++w) {
                        f[x] += sm.part[x][w][e];
                        sm.part[x][w][e] = 0.0f;
                    }
                const uint32_t g = sm.gid[b][e];
                if (f[0] != 0.0f) atomicAdd(a.afg + g, f[0]);
                if (f[1] != 0.0f) atomicAdd(a.abg + g, f[1]);
            } else if (!kReal && e < cnt) {
                const uint32_t g = sm.gid[b][e];
                const uint32_t v0 = sm.acc0[b][e];
                if (v0) {
                    atomicAdd((MODE == 1 ? a.resp : a.fg) + g, v0);
                    sm.acc0[b][e] = 0u;
                }
                if (MODE == 2) {
                    const uint32_t v1 = sm.acc1[b][e];
                    if (v1) {
                        atomicAdd(a.bg + g, v1);
                        sm.acc1[b][e] = 0u;
                    }
                }
            }
        }
    };
    // Mode 3: whether this warp's pixels lie on both sides of the mask, else
    // which side they are on.
    const bool mixed = kReal && !__all_sync(0xffffffffu, inside) && __any_sync(0xffffffffu, inside);
    const uint32_t side = kReal && inside ? 0u : 1u;
    const f32x2 nfx = both(-fx), nfy = both(-fy);
    auto* const recs = sm.pairs[warp];
    auto done = [&]() { return ps.T < inv255; };

    // Composites one entry into this lane's pixel: npow = -power, e =
    // exp(npow); returns alpha T where the entry contributes (the pixel is not
    // saturated, T >= 1/255; alpha >= 1/255; power no higher than power_max or
    // NaN), else 0. Written with predicates: as branches, the two entries of a
    // pair cost a third more instructions.
    auto composite = [&](float npow, float npm, float op, float e, float cr, float cg, float cb,
                         uint32_t pos) -> float {
        const float alpha = fminf(op * e, 0.999f);
        float vis;
        if (DETAIL) {
            const bool eval = ps.T >= inv255 && !(npow < npm);
            ps.n_eval += eval;
            ps.n_hit += eval && alpha >= inv255;
        }
        const float t0 = ps.T;
        if constexpr (kColor) {
            asm("{\n"
                ".reg .pred p;\n"
                ".reg .f32 m;\n"
                "setp.ge.f32 p, %0, %5;\n"
                "setp.ge.and.f32 p, %6, %5, p;\n"
                "setp.geu.and.f32 p, %7, %8, p;\n"
                "mul.rn.f32 %4, %6, %0;\n"
                "sub.rn.f32 m, 0f3F800000, %6;\n"
                "@p fma.rn.f32 %1, %9, %4, %1;\n"
                "@p fma.rn.f32 %2, %10, %4, %2;\n"
                "@p fma.rn.f32 %3, %11, %4, %3;\n"
                "@p mul.rn.f32 %0, %0, m;\n"
                "}"
                : "+f"(ps.T), "+f"(ps.pr), "+f"(ps.pg), "+f"(ps.pb), "=&f"(vis)
                : "f"(inv255), "f"(alpha), "f"(npow), "f"(npm), "f"(cr), "f"(cg), "f"(cb));
        } else {
            asm("{\n"
                ".reg .pred p;\n"
                ".reg .f32 m;\n"
                "setp.ge.f32 p, %0, %2;\n"
                "setp.ge.and.f32 p, %3, %2, p;\n"
                "setp.geu.and.f32 p, %4, %5, p;\n"
                "mul.rn.f32 %1, %3, %0;\n"
                "sub.rn.f32 m, 0f3F800000, %3;\n"
                "selp.f32 %1, %1, 0f00000000, p;\n"
                "@p mul.rn.f32 %0, %0, m;\n"
                "}"
                : "+f"(ps.T), "=&f"(vis)
                : "f"(inv255), "f"(alpha), "f"(npow), "f"(npm));
        }
        if (EXACT && ps.T != t0) ps.last = pos;  // T always falls where the entry contributes
        return vis;
    };
    // The warp's 32 shares of entry j to its shared accumulators.
    auto add_words = [&](uint32_t q, uint32_t b, uint32_t j) {
        if (!__any_sync(0xffffffffu, q != 0u)) return;
        if (MODE == 1) {
            const uint32_t s = __reduce_add_sync(0xffffffffu, q);
            if (lane == 0) atomicAdd(&sm.acc0[b][j], s);
        } else {
            const uint32_t qf = inside ? q : 0u;
            const uint32_t sf = __reduce_add_sync(0xffffffffu, qf);
            const uint32_t st = __reduce_add_sync(0xffffffffu, q);
            if (lane == 0) {
                if (sf) atomicAdd(&sm.acc0[b][j], sf);
                if (st - sf) atomicAdd(&sm.acc1[b][j], st - sf);
            }
        }
    };
    // The two entries of recs[p]: both alphas by packed operations, then the
    // pixel takes them in order. Every lane of the warp runs it together.
    auto step2 = [&](uint32_t p, uint32_t b, uint32_t pos0, float& wa, float& wb, uint32_t& ja, uint32_t& jb) {
        const float4* r4 = reinterpret_cast<const float4*>(recs + p);
        const ulonglong2* r = reinterpret_cast<const ulonglong2*>(recs + p);
        const ulonglong2 xy = r[0], hc = r[1], zo = r[2];
        const float4 mj = r4[3];
        float4 rg = make_float4(0.f, 0.f, 0.f, 0.f);
        float2 bl = make_float2(0.f, 0.f);
        if (kColor) {
            rg = r4[4];
            bl = *reinterpret_cast<const float2*>(r4 + 5);
        }
        ja = f2u(mj.z);
        jb = f2u(mj.w);
        const f32x2 dx = add2(xy.x, nfx), dy = add2(xy.y, nfy);
        const f32x2 npow = fma2(mul2(hc.x, dx), dx, fma2(mul2(zo.x, dy), dy, mul2(mul2(hc.y, dx), dy)));
        float na, nb, oa, ob, ea, eb;
        exp_neg2(npow, ea, eb);
        unpack2(npow, na, nb);
        unpack2(zo.y, oa, ob);
        wa = composite(na, mj.x, oa, ea, rg.x, rg.z, bl.x, pos0 + ja);
        wb = composite(nb, mj.y, ob, eb, rg.y, rg.w, bl.y, pos0 + jb);
        if (kWords) {
            add_words(sat_u32(wa * a.scale), b, ja);
            add_words(sat_u32(wb * a.scale), b, jb);
        }
    };
    // Up to 32 candidates [g32, g32 + 32) of buffer b, of which this lane's is
    // walked when `hit`: the hits are packed two by two into recs in list
    // order (an odd last one beside an entry that no pixel takes) and
    // composited.
    auto walk = [&](uint32_t b, uint32_t g32, bool hit, const float4& g0, const float4& g1, uint32_t pos0) {
        const uint32_t word = __ballot_sync(0xffffffffu, hit);
        const uint32_t hits = (uint32_t)__popc(word);
        if (hits == 0) return;
        if (DETAIL) ps.n_proc += hits;
        __syncwarp();  // the last group's records have been read
        if (hit) {
            const uint32_t slot = (uint32_t)__popc(word & ((1u << lane) - 1u)), h = slot & 1u;
            auto& r = recs[slot >> 1];
            if (kColor) {
                const float4 c = sm.col[b][g32 + lane];
                r.r[h] = c.x;
                r.g[h] = c.y;
                r.b[h] = c.z;
            }
            r.x[h] = g0.x;
            r.y[h] = g0.y;
            r.nhx[h] = -g0.z;
            r.ncy[h] = -g0.w;
            r.nhz[h] = -g1.x;
            r.op[h] = g1.y;
            r.npm[h] = -g1.z;
            r.j[h] = g32 + lane;
        }
        if ((hits & 1u) && lane == 0) {
            auto& r = recs[hits >> 1];
            r.x[1] = r.y[1] = r.nhx[1] = r.ncy[1] = r.nhz[1] = r.op[1] = 0.0f;
            r.npm[1] = INFINITY;  // past every power: not an evaluated pair either
            if (kColor) r.r[1] = r.g[1] = r.b[1] = 0.0f;
            r.j[1] = g32;
        }
        __syncwarp();
        const uint32_t np = (hits + 1u) >> 1;
        if constexpr (!kReal) {
            float wa, wb;
            uint32_t ja, jb;
            for (uint32_t p = 0; p < np; ++p) step2(p, b, pos0, wa, wb, ja, jb);
        } else {
            // Mode 3: four entries' weights are summed over the warp at once.
            const uint32_t which = mixed ? (lane >> 2) & 3u : lane >> 3;
            for (uint32_t p = 0; p < np; p += 2) {
                float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                uint32_t j[4] = {0u, 0u, 0u, 0u};
                step2(p, b, pos0, v[0], v[1], j[0], j[1]);
                if (p + 1 < np) step2(p + 1, b, pos0, v[2], v[3], j[2], j[3]);
                const float any = fmaxf(fmaxf(v[0], v[1]), fmaxf(v[2], v[3]));
                if (!__any_sync(0xffffffffu, any != 0.0f)) continue;
                // The entry whose sum this lane ends with.
                const uint32_t mine = which < 2 ? (which == 0 ? j[0] : j[1]) : (which == 2 ? j[2] : j[3]);
                if (mixed) {
                    float x[8];
#pragma unroll
                    for (uint32_t u = 0; u < 4; ++u) {
                        x[u] = inside ? v[u] : 0.0f;
                        x[4 + u] = inside ? 0.0f : v[u];
                    }
                    warp_sum_scatter(x);
                    if ((lane & 3u) == 0 && x[0] != 0.0f) sm.part[lane >> 4][warp][mine] = x[0];
                } else {
                    warp_sum_scatter(v);
                    if ((lane & 7u) == 0 && v[0] != 0.0f) sm.part[side][warp][mine] = v[0];
                }
            }
        }
    };

    load_ids(0);
    issue(0, 0);
    cp_async_commit();
    if (nchunks > 1) load_ids(1);
    for (uint32_t c = 0; c < nchunks; ++c) {
        const uint32_t b = c & 1u;
        cp_async_wait<0>();  // this thread's copies of chunk c have landed
        // One barrier: every thread's copies of chunk c are there, and the
        // walk of chunk c - 1 is over, so its sums are complete and its buffer
        // may be refilled.
        const bool all_done = __syncthreads_count(done()) == NT;
        if ((kWords || kReal) && c > 0) flush(b ^ 1u, kChunk);
        if (all_done) return true;
        if (c + 1 < nchunks) {
            issue(c + 1, b ^ 1u);
            cp_async_commit();
            if (c + 2 < nchunks) load_ids(c + 2);
        }
        if (kReal) __syncthreads();  // the warps' sums of the last chunk have been read
        const uint32_t cnt = min(kChunk, count - c * kChunk);
        if (!EXACT && !done()) ps.last = c * kChunk + cnt;
        const uint32_t pos0 = list_off + c * kChunk + 1;
        for (uint32_t g32 = 0; g32 < cnt; g32 += 32) {
            if (__all_sync(0xffffffffu, done())) break;
            const uint32_t j = g32 + lane;
            bool hit = j < cnt;
            float4 g0 = make_float4(0.f, 0.f, 0.f, 0.f), g1 = g0;
            if (hit) {
                g0 = sm.g0[b][j];
                g1 = sm.g1[b][j];
                if (CULL) hit = block_hit(g0, g1, sm.ext[b][j], wxf, wyf);
            }
            walk(b, g32, hit, g0, g1, pos0);
        }
    }
    __syncthreads();
    if (kWords || kReal) flush((nchunks - 1) & 1u, count - (nchunks - 1) * kChunk);
    return false;
}

__device__ __forceinline__ unsigned long long pair_value(uint2 p) {
    return ((unsigned long long)p.x << 32) | p.y;
}

// Block min / max of 64-bit values (uniform); s64 holds 2 * 8 words.
template <uint32_t NT>
__device__ void block_minmax64(unsigned long long lo, unsigned long long hi, unsigned long long* s64,
                               unsigned long long& mn, unsigned long long& mx) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
#pragma unroll
    for (uint32_t d = 16; d > 0; d >>= 1) {
        lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, d));
        hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, d));
    }
    __syncthreads();
    if (lane == 0) {
        s64[warp] = lo;
        s64[8 + warp] = hi;
    }
    __syncthreads();
    mn = s64[0];
    mx = s64[8];
    for (uint32_t w = 1; w < NT / 32; ++w) {
        mn = min(mn, s64[w]);
        mx = max(mx, s64[8 + w]);
    }
    __syncthreads();
}

// Bitonic sort of v[0, m) ascending in shared memory (m <= kSlab), padded to
// a power of two with the largest value.
template <uint32_t NT>
__device__ void bitonic_sort64(unsigned long long* v, uint32_t m) {
    uint32_t p = 1;
    while (p < m) p <<= 1;
    for (uint32_t i = m + threadIdx.x; i < p; i += NT) v[i] = ~0ull;
    __syncthreads();
    for (uint32_t k = 2; k <= p; k <<= 1) {
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            for (uint32_t i = threadIdx.x; i < p; i += NT) {
                const uint32_t ixj = i ^ j;
                if (ixj > i) {
                    const unsigned long long x = v[i], y = v[ixj];
                    const bool up = (i & k) == 0;
                    if ((x > y) == up) {
                        v[i] = y;
                        v[ixj] = x;
                    }
                }
            }
            __syncthreads();
        }
    }
}

// Shared memory of one CTA.
template <int MODE, bool CULL, bool LAZY, uint32_t NT>
struct TileShared {
    Stage<MODE, CULL, NT> stage;
    unsigned long long slab[LAZY ? kSlab : 1];
    unsigned long long s64[16];
    uint32_t hist[LAZY ? 256 : 1];
    uint32_t ctl[4];
};

// This CTA's part `sub` of one tile (block-uniform).
// TAIL: the tile's tail, from the transmittances that its head left.
template <int MODE, bool CULL, bool DETAIL, bool STATE, bool LAZY, bool TAIL, uint32_t NT>
__device__ __forceinline__ void raster_tile(const RasterArgs& a, const uint32_t tile, const uint32_t sub) {
    extern __shared__ __align__(16) unsigned char s_tile[];
    TileShared<MODE, CULL, LAZY, NT>& sh = *reinterpret_cast<TileShared<MODE, CULL, LAZY, NT>*>(s_tile);
    Stage<MODE, CULL, NT>& sm = sh.stage;
    unsigned long long* const s_slab = sh.slab;
    uint32_t* const s_hist = sh.hist;
    unsigned long long* const s_64 = sh.s64;
    uint32_t* const s_ctl = sh.ctl;

    const uint32_t tx = tile % a.tiles_x, ty = tile / a.tiles_x;
    const uint32_t tid = threadIdx.x, lane = tid & 31u;
    const uint32_t wt = sub * (NT / 32) + (tid >> 5);  // warp of the tile
    const uint32_t wx0 = tx * 16 + (wt & 1u) * 8, wy0 = ty * 16 + (wt >> 1) * 4;
    const uint32_t px = wx0 + (lane & 7u);
    const uint32_t py = wy0 + (lane >> 3);
    const bool in_bounds = px < a.w && py < a.h;
    const float fx = (float)px + 0.5f, fy = (float)py + 0.5f;
    const float wxf = (float)wx0 + 0.5f, wyf = (float)wy0 + 0.5f;
    uint32_t inside = 0;
    if (MODE == 3) inside = !a.mask || !in_bounds;  // pixels outside the image weigh nothing
    if ((MODE == 2 || (MODE == 3 && a.mask)) && in_bounds) inside = (a.mask[px / 32 + py * a.mask_wpr] >> (px % 32)) & 1u;
    const uint32_t start = TAIL ? a.tail_start[tile] : a.tile_start[tile];
    const uint32_t end = TAIL ? start + a.tail_n[tile] : a.tile_start[tile + 1];
    // A pixel takes entries while T >= 1/255; those outside the image start done.
    PixelState ps{!in_bounds ? 0.0f : TAIL ? a.head_t[(size_t)py * a.w + px] : 1.0f, 0.0f, 0.0f, 0.0f, 0u, 0u, 0u, 0u};
    if (ModeOf<MODE>::kWords) {
        for (uint32_t e = tid; e < kChunk; e += NT) {
            sm.acc0[0][e] = sm.acc0[1][e] = 0u;
            if (MODE == 2) sm.acc1[0][e] = sm.acc1[1][e] = 0u;
        }
    }
    if (ModeOf<MODE>::kReal) {
        for (uint32_t e = tid; e < 2 * (NT / 32) * kChunk; e += NT)
            sm.part[e / ((NT / 32) * kChunk)][e / kChunk % (NT / 32)][e % kChunk] = 0.0f;
    }

    if (!LAZY || end - start <= a.lazy_min) {
        const uint32_t* ids = a.gaussian_ids + start;
        composite_list<MODE, CULL, DETAIL, STATE || LAZY, NT>(
            a, sm, [&](uint32_t i) { return __ldg(ids + i); }, end - start, 0, fx, fy, wxf, wyf, inside, ps);
    } else if (end > start) {
        const uint2* pairs = a.pairs + start;
        const uint32_t n = end - start;
        unsigned long long lo = ~0ull, hi = 0;
        for (uint32_t i = tid; i < n; i += NT) {
            const unsigned long long v = pair_value(pairs[i]);
            lo = min(lo, v);
            hi = max(hi, v);
        }
        unsigned long long vmin, vmax;
        block_minmax64<NT>(lo, hi, s_64, vmin, vmax);
        auto slab_id = [&](uint32_t i) { return (uint32_t)s_slab[i]; };
        if (n <= kFirstSlab) {
            for (uint32_t i = tid; i < n; i += NT) s_slab[i] = pair_value(pairs[i]);
            __syncthreads();
            bitonic_sort64<NT>(s_slab, n);
            composite_list<MODE, CULL, DETAIL, STATE || LAZY, NT>(a, sm, slab_id, n, 0, fx, fy, wxf, wyf, inside, ps);
        } else {
            unsigned long long cur = vmin;
            uint32_t pos = 0;
            // The first slab aims at kFirstSlab entries (most tiles saturate
            // well inside it), later ones at the full kSlab.
            uint32_t target = TAIL ? kSlab : kFirstSlab;
            for (;;) {
                // Pick [cur, sel] holding at most `target` of the values left
                // (one whole bin of up to kSlab when the first bin alone is
                // past the target).
                unsigned long long top = vmax, sel = vmax;
                for (;;) {
                    const unsigned long long width = top - cur;
                    const uint32_t wbits = width == 0 ? 0u : 64u - (uint32_t)__clzll(width);
                    const uint32_t shift = wbits > 8 ? wbits - 8 : 0u;
                    for (uint32_t i = tid; i < 256; i += NT) s_hist[i] = 0;
                    __syncthreads();
                    for (uint32_t i = tid; i < n; i += NT) {
                        const unsigned long long v = pair_value(pairs[i]);
                        if (v >= cur && v <= top) atomicAdd(&s_hist[(uint32_t)((v - cur) >> shift)], 1u);
                    }
                    __syncthreads();
                    if (tid < 32) {
                        // Warp 0: prefix over the 256 bins (8 per lane), the
                        // last bin whose running total stays within target.
                        const uint32_t nb = (uint32_t)(width >> shift) + 1u;
                        uint32_t c[8], run = 0;
#pragma unroll
                        for (uint32_t q = 0; q < 8; ++q) {
                            const uint32_t bn = lane * 8 + q;
                            c[q] = bn < nb ? s_hist[bn] : 0u;
                            run += c[q];
                        }
                        uint32_t incl = run;
#pragma unroll
                        for (uint32_t d = 1; d < 32; d <<= 1) {
                            const uint32_t x = __shfl_up_sync(0xffffffffu, incl, d);
                            if (lane >= d) incl += x;
                        }
                        uint32_t acc = incl - run, best = 0u;
                        bool any = false;
#pragma unroll
                        for (uint32_t q = 0; q < 8; ++q) {
                            acc += c[q];
                            const uint32_t bn = lane * 8 + q;
                            if (bn < nb && acc <= target) {
                                best = bn;
                                any = true;
                            }
                        }
                        const uint32_t e = __reduce_max_sync(0xffffffffu, any ? best + 1u : 0u);
                        if (lane == 0) {
                            const uint32_t h0 = s_hist[0];
                            // e == 0: even bin 0 is past the target.
                            s_ctl[0] = e > 0 ? 1u : (h0 <= kSlab ? 1u : 0u);
                            s_ctl[1] = e > 0 ? e - 1u : 0u;
                            s_ctl[2] = nb;
                        }
                    }
                    __syncthreads();
                    const uint32_t e = s_ctl[1], bins = s_ctl[2];
                    if (!s_ctl[0]) {
                        // The first bin holds more than kSlab: narrow to it.
                        top = cur + ((1ull << shift) - 1ull);
                        continue;
                    }
                    sel = (e + 1 >= bins) ? top : cur + (((unsigned long long)(e + 1)) << shift) - 1ull;
                    break;
                }
                if (tid == 0) s_ctl[3] = 0;
                __syncthreads();
                for (uint32_t i = tid; i < n; i += NT) {
                    const unsigned long long v = pair_value(pairs[i]);
                    if (v >= cur && v <= sel) s_slab[atomicAdd(&s_ctl[3], 1u)] = v;
                }
                __syncthreads();
                const uint32_t m = s_ctl[3];
                bitonic_sort64<NT>(s_slab, m);
                if (composite_list<MODE, CULL, DETAIL, STATE || LAZY, NT>(a, sm, slab_id, m, pos, fx, fy, wxf, wyf,
                                                                  inside, ps))
                    break;
                pos += m;
                if (sel == vmax) break;
                cur = sel + 1;
                target = kSlab;
                __syncthreads();
            }
        }
    }
    if (MODE != 0 && !TAIL && a.head_limit && a.head_limit[tile] != 0xffffffffu) {
        // A head with a tail behind it: the transmittances are kept, and the
        // tile is listed when one of this CTA's pixels takes more entries.
        if (in_bounds) a.head_t[(size_t)py * a.w + px] = ps.T;
        if (__syncthreads_or(ps.T >= 1.0f / 255.0f) && tid == 0) {
            const uint32_t bit = 1u << (tile & 31u);
            if (!(atomicOr(a.head_bits + (tile >> 5), bit) & bit)) a.head_list[atomicAdd(a.head_ctrl, 1u)] = tile;
        }
    }
    if (a.stats) {
        if (DETAIL) {
            const uint32_t e = __reduce_add_sync(0xffffffffu, ps.n_eval);
            const uint32_t c = __reduce_add_sync(0xffffffffu, ps.n_hit);
            const uint32_t pr_ = __reduce_add_sync(0xffffffffu, ps.n_proc);
            if (lane == 0) {
                atomicAdd(a.stats + 1, (unsigned long long)e);
                atomicAdd(a.stats + 2, (unsigned long long)c);
                atomicAdd(a.stats + 3, (unsigned long long)pr_);
            }
        }
        // Algorithmic pairs: this CTA's pixels times the entries of the
        // sorted list that a walk in 256-entry chunks covers until every one
        // of them is saturated — the entry that saturates its last pixel,
        // rounded up to a chunk (the whole list if a pixel never saturates).
        // With one CTA per tile, 256 per entry the tile walks. The same
        // count for either list order.
        const uint32_t n_list = end - start;
        uint32_t e = ps.T < 1.0f / 255.0f ? ps.last : n_list;
        e = __reduce_max_sync(0xffffffffu, e);
        __syncthreads();
        if (tid == 0) s_ctl[0] = 0;
        __syncthreads();
        if (lane == 0) atomicMax(&s_ctl[0], e);
        __syncthreads();
        if (tid == 0) {
            const uint32_t emax = s_ctl[0];
            const uint64_t chunks = ((uint64_t)emax + kChunk - 1) / kChunk * kChunk;
            const uint64_t walked = chunks < n_list ? chunks : (uint64_t)n_list;
            atomicAdd(a.stats, (unsigned long long)NT * walked);
        }
    }
    if (!in_bounds) return;
    const size_t pix = (size_t)py * a.w + px;
    if (MODE == 0) {
        if (a.bitmap) {
            const uint32_t r = sat_u32(clamp_(ps.pr * 255.0f, 0.0f, 255.0f));
            const uint32_t g = sat_u32(clamp_(ps.pg * 255.0f, 0.0f, 255.0f));
            const uint32_t b = sat_u32(clamp_(ps.pb * 255.0f, 0.0f, 255.0f));
            const uint32_t al = sat_u32(clamp_((1.0f - ps.T) * 255.0f, 0.0f, 255.0f));
            a.bitmap[(size_t)py * a.row_stride + px] = r | (g << 8) | (b << 16) | (al << 24);
        }
        if (a.rgba) a.rgba[pix] = make_float4(ps.pr, ps.pg, ps.pb, 1.0f - ps.T);
    }
    if (STATE) {
        if (a.final_t) a.final_t[pix] = ps.T;
        if (a.n_contrib) a.n_contrib[pix] = ps.last;
    }
}

// 256 / NT CTAs per tile: block i takes part i % (256 / NT) of tile i /
// (256 / NT), or with class lists of the tile of that rank in longest-list-
// first order.
template <int MODE, bool CULL, bool DETAIL, bool STATE, bool LAZY, uint32_t NT>
__global__ __launch_bounds__(NT) void raster_kernel(RasterArgs a) {
    constexpr uint32_t kSplit = 256 / NT;
    const uint32_t rank = blockIdx.x / kSplit, sub = blockIdx.x % kSplit;
    uint32_t tile = rank;
    if (a.class_lists) {
        const uint32_t tiles = a.tiles_x * a.tiles_y;
        uint32_t j = rank;
        int k = kSortClasses - 1;
        for (; k >= 0; --k) {
            const uint32_t c = a.class_n[k];
            if (j < c) break;
            j -= c;
        }
        // k < 0: the empty tiles (the counts sum to the tile count).
        tile = a.class_lists[(size_t)(k < 0 ? kSortClasses : k) * tiles + j];
    }
    raster_tile<MODE, CULL, DETAIL, STATE, LAZY, false, NT>(a, tile, sub);
}

// The tails of the listed tiles, a CTA each in turn.
template <int MODE>
__global__ __launch_bounds__(256) void raster_tails_kernel(RasterArgs a) {
    const uint32_t count = a.head_ctrl[1] ? 0u : a.head_ctrl[0];
    for (uint32_t i = blockIdx.x; i < count; i += gridDim.x) {
        raster_tile<MODE, true, false, false, true, true, 256>(a, a.head_list[i], 0);
        __syncthreads();
    }
}

template <int MODE, bool CULL, bool DETAIL, bool STATE, bool LAZY, uint32_t NT>
cudaError_t raster_go(const RasterArgs& a, uint32_t tiles, cudaStream_t st) {
    constexpr size_t smem = sizeof(TileShared<MODE, CULL, LAZY, NT>);
    auto kernel = raster_kernel<MODE, CULL, DETAIL, STATE, LAZY, NT>;
    if (smem > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    kernel<<<tiles * (256 / NT), NT, smem, st>>>(a);
    return cudaGetLastError();
}

template <int MODE, bool LAZY>
cudaError_t raster_dispatch(const RasterArgs& a, uint32_t tiles, cudaStream_t st) {
    // The per-pixel state (for the adjoint, and in mode 3 for read-backs of
    // the frame) and the pair diagnostics are kept by one CTA per tile.
    constexpr bool kState = MODE == 0 || MODE == 3;
    if (a.detail) {
        return a.cull ? raster_go<MODE, true, true, kState, LAZY, 256>(a, tiles, st)
                      : raster_go<MODE, false, true, kState, LAZY, 256>(a, tiles, st);
    }
    if (kState && (a.final_t || a.n_contrib)) return raster_go<MODE, true, false, kState, LAZY, 256>(a, tiles, st);
    if (a.split == 4) return raster_go<MODE, true, false, false, LAZY, 64>(a, tiles, st);
    if (a.split == 2) return raster_go<MODE, true, false, false, LAZY, 128>(a, tiles, st);
    return raster_go<MODE, true, false, false, LAZY, 256>(a, tiles, st);
}

template <int MODE>
cudaError_t tails_go(const RasterArgs& a, int sm_count, cudaStream_t st) {
    constexpr size_t smem = sizeof(TileShared<MODE, true, true, 256>);
    if (smem > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(raster_tails_kernel<MODE>,
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    const uint32_t tiles = a.tiles_x * a.tiles_y;
    raster_tails_kernel<MODE><<<std::min(tiles, 3u * (uint32_t)std::max(sm_count, 1)), 256, smem, st>>>(a);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_raster(int mode, const RasterArgs& args, cudaStream_t stream) {
    const uint32_t tiles = args.tiles_x * args.tiles_y;
    if (tiles == 0) return cudaSuccess;
    RasterArgs a = args;
    if (a.split == 0) a.split = 1;
    if (a.split != 1 && a.split != 2 && a.split != 4) return cudaErrorInvalidValue;
    if (!a.ext) return cudaErrorInvalidValue;
    const bool lazy = a.pairs != nullptr;
    cudaError_t e = cudaErrorInvalidValue;
    switch (mode) {
        case 0: e = lazy ? raster_dispatch<0, true>(a, tiles, stream) : raster_dispatch<0, false>(a, tiles, stream); break;
        case 1: e = lazy ? raster_dispatch<1, true>(a, tiles, stream) : raster_dispatch<1, false>(a, tiles, stream); break;
        case 2: e = lazy ? raster_dispatch<2, true>(a, tiles, stream) : raster_dispatch<2, false>(a, tiles, stream); break;
        case 3:
            if (a.afg && a.abg && !lazy) e = raster_dispatch<3, false>(a, tiles, stream);
            break;
        default: break;
    }
    if (e == cudaSuccess) note_launches(1);
    return e;
}

cudaError_t launch_raster_tails(int mode, const RasterArgs& args, int sm_count, cudaStream_t stream) {
    RasterArgs a = args;
    a.lazy_min = 0;
    a.stats = nullptr;
    if (!a.pairs || !a.ext || !a.tail_start || !a.tail_n || !a.head_ctrl || !a.head_list || !a.head_t)
        return cudaErrorInvalidValue;
    cudaError_t e = cudaErrorInvalidValue;
    switch (mode) {
        case 1: e = tails_go<1>(a, sm_count, stream); break;
        case 2: e = tails_go<2>(a, sm_count, stream); break;
        case 3: e = tails_go<3>(a, sm_count, stream); break;
        default: break;
    }
    if (e == cudaSuccess) note_launches(1);
    return e;
}

}  // namespace sfk
