// Handle types shared by the C ABI translation units (sf_api.cu, sf_round.cu).
#pragma once
#include <atomic>
#include <cstdint>
#include <mutex>
#include <string>
#include "sf_internal.h"

// One number per handle made, never given twice. Captured graphs keep it to
// tell the handle they were captured with from a later one at its address,
// whose device buffers are others.
inline uint64_t next_handle_id() {
    static std::atomic<uint64_t> next{1};
    return next.fetch_add(1, std::memory_order_relaxed);
}

struct sf_ctx_t {
    int device = 0;
    int sm_count = 148;
    float* lut = nullptr;  // f32 entropy LUT, built on first use
    // Page-locked error words of the sort and scan scratches: one page, taken
    // by the first of them and held until the context goes (page-locking costs
    // a millisecond or more, a whole scratch 0.4). word_used: a bit per slot.
    std::mutex word_mu;
    uint32_t* word_page = nullptr;
    uint64_t word_used = 0;
};

struct sf_splats_t {
    const uint64_t id = next_handle_id();
    sf_ctx ctx = nullptr;
    uint32_t n = 0, K = 1;
    float* attr = nullptr;
    float* sh = nullptr;
    float* geom = nullptr;  // [kGeomPlanes][n] camera-independent projection terms of attr
    float bounds[6] = {0, 0, 0, 0, 0, 0};
};

struct sf_accum_t {
    sf_ctx ctx = nullptr;
    uint32_t total = 0;
    uint32_t *resp = nullptr, *fg = nullptr, *bg = nullptr;
    float scale = 1.0f;
    bool evidence = false;  // the last fill was a masked split (fg, bg), not resp
};

struct sf_mask_t {
    const uint64_t id = next_handle_id();
    uint32_t w = 0, h = 0, wpr = 0;
    uint32_t* bits = nullptr;
};

struct sf_beta_t {
    const uint64_t id = next_handle_id();
    sf_ctx ctx = nullptr;
    uint32_t n = 0;
    float *a = nullptr, *b = nullptr;
    double* partials = nullptr;
    uint32_t blocks = 1;
    double* host_out = nullptr;  // pinned; the last kernel of a synchronous EIG writes it
    // Localization scratch (allocated on first use): [blocks][4] partials,
    // [8] results, pinned mirror of the results.
    double* loc_partials = nullptr;
    double* loc_out = nullptr;
    double* loc_host = nullptr;
};

namespace sfk {
// Records the calling thread's last error message (sf_last_error) and
// returns `code`.
int set_error(int code, const std::string& msg);
}  // namespace sfk
