// abi.cu -- the C ABI of libgb300ntt.so (declared in include/gb300_ntt.h).
#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <new>
#include <string>

#include "../../include/gb300_ntt.h"
#include "batch_kernel.cuh"
#include "canon_tables.h"
#include "device.cuh"
#include "plan_internal.h"
#include "tables.h"
#include "tc16.cuh"

namespace gbntt {
const void* bitrev_kernel_ptr();
const void* tc16_kernel(int L, bool bitrev_in, bool bitrev_out);   // kernels_tc16.cu
}

using namespace gbntt;

struct gbntt_plan {
    HostPlan hp;
    int fam = -1;          // transform family of k_ntt, -1 for the single-purpose kernels
    bool br = false;       // bit-reversed load and store (radix-4 inverse)
    KernelInfo ki;
    KernelInfo kl;         // latency form for launches of at most one CTA per SM (fn nullptr: none)
    LargeInfo large;       // int32 n >= 2^14: two-pass schedule (large.cols != nullptr)
    CanonLarge clarge;     // canonical int32 n >= 2^14: two passes (clarge.cols != nullptr)
    uint64_t two_pass_max = 0;        // calls of more polynomials than this run one CTA per polynomial
    const int2* tab_blocks = nullptr; // clarge: the tables of the two passes (inside d_tab)
    unsigned* d_err = nullptr;        // clarge: set when a bounded wait ran out
    KArgs base;            // constants shared by every launch
    int2* d_tab = nullptr;
    size_t tab_bytes = 0;
    size_t tile_tab_bytes = 0;   // of these, the table of the one-CTA kernels (first in d_tab)
    size_t tc_bytes = 0;   // tensor-core table behind it in the same allocation
    const void* tc_fn = nullptr;   // tensor-core kernel (canonical int16, n = 2^6 .. 2^10)
    int device = 0;
    std::mutex stage_mu;   // serialises gbntt_execute_host on this plan
    void* d_stage = nullptr;
    size_t stage_bytes = 0;
    void* zc_state = nullptr;   // zero-copy scratch (batch.cu), created on first use
};

namespace {

thread_local std::string g_err;
std::atomic<unsigned long long> g_launches{0};

int fail(int code, const std::string& msg) {
    g_err = msg;
    return code;
}

int cuda_fail(cudaError_t e, const char* what) {
    g_err = std::string(what) + ": " + cudaGetErrorString(e);
    return GBNTT_ERR_CUDA;
}

int family_of(int kind) {
    switch (kind) {
    case K_R2_I16_FWD: return F_R2F16;
    case K_R2_I16_INV: return F_R2I16;
    case K_R4_I16_FWD: return F_R4F16;
    case K_R4_I16_INV: return F_R4F16;
    case K_R8_I16_FWD: return F_R8F16;
    case K_R2_I32_FWD: return F_R2F32;
    case K_R2_I32_INV: return F_R2G32;
    default: return -1;
    }
}

KernelInfo kernel_for(int fam, int L, bool br, bool lat, int form) {
    if (fam_canon(fam)) return kinfo_canon(fam, L, lat);
    switch (fam) {
    case F_R2F16: return kinfo_r2f16(L, lat, form);
    case F_R2I16: return kinfo_r2i16(L, lat, form);
    case F_R4F16: return kinfo_r4(L, br, lat);
    case F_R8F16: return kinfo_r8(L, lat);
    case F_R2F32: return kinfo_r2f32(L, lat);
    case F_R2G32: return kinfo_r2g32(L, lat);
    default: return KernelInfo();
    }
}

int sm_count() {
    static const int sms = [] {
        int dev = 0, n = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        return n > 0 ? n : 1;
    }();
    return sms;
}

// The largest call, in polynomials, that an int32 plan of 2^L coefficients
// runs in two passes (0: none, UINT64_MAX: every one); 2^14 and 2^15 also fit
// one CTA per polynomial, 2^16 and more do not.  One CTA takes the same time
// for 1 polynomial as for 152 and keeps half an SM's threads waiting at its
// barriers; two passes spread a polynomial over 16 .. 64 CTAs.  Measured (us,
// one CTA -> two passes; 1 / 76 / 152 / 1024 / 2^26 n^-1 polynomials):
//   canonical 2^14 forward  15.0 / 15.0 / 17.0 / 58 / 193 -> 10.9 / 12.9 / 17.0 / 59 / 204
//   canonical 2^14 inverse  15.0 / 15.0 / 17.0 / 60 / 197 -> 8.8 / 11.9 / 16.0 / 54 / 189
//   canonical 2^15          21.1 / 23.2 / 25.2 / 127 / 240 -> 10.9 / 17.0 / 25.2 / 107 / 197
//   lanes 2^14              18.0 / 19.0 / 19.1 / 85 / 302 -> 10.9 / 16.0 / 21.1 / 88 / 323
//   lanes 2^15              33.4 / 33.4 / 35.5 / 196 / 388 -> 10.9 / 22.1 / 33.4 / 168 / 321
// so 2^15 and the canonical inverse of 2^14 always take two passes and the
// others of 2^14 up to half a polynomial per SM.  GBNTT_FOURSTEP_MIN_L (14 .. 16,
// read once per process) instead runs canonical lengths from 2^that on in two
// passes and shorter ones in one CTA.
uint64_t two_pass_limit(int L, bool canon, bool inverse) {
    static const int env = [] {
        const char* e = std::getenv("GBNTT_FOURSTEP_MIN_L");
        const int x = e ? std::atoi(e) : 0;
        return x >= 14 && x <= 16 ? x : 0;
    }();
    if (L < 14) return 0;
    if (L >= 16) return UINT64_MAX;
    if (canon && env) return L >= env ? UINT64_MAX : 0;
    return L == 15 || (canon && inverse) ? UINT64_MAX : (uint64_t)(sm_count() / 2);
}

int launch(const gbntt_plan* p, const void* d_in, void* d_out, uint64_t batch, cudaStream_t s) {
    KArgs a = p->base;
    a.in = d_in;
    a.out = d_out;
    a.batch = (long long)batch;
    cudaError_t e = cudaSuccess;
    // a call whose grid would not fit one launch is refused, whatever form it takes
    auto too_large = [&](unsigned long long blocks_per_poly) { return batch > 0x7FFFFFFFull / blocks_per_poly; };
    if (p->clarge.cols && batch <= p->two_pass_max) {
        const CanonLarge& li = p->clarge;
        if (too_large(std::max(1ull << li.L1, (1ull << li.L2) / li.cols_width)))
            return fail(GBNTT_ERR_ARG, "batch too large for one launch");
        const bool inverse = (p->hp.kind == K_R2_I32_INV);
        int nl = 0;
        e = launch_canon_large(li, a, p->tab_blocks, d_in, d_out, (long long)batch, inverse, p->d_err, s, &nl);
        if (e != cudaSuccess) return cuda_fail(e, "two-pass launch");
        g_launches.fetch_add((unsigned long long)nl, std::memory_order_relaxed);
        return GBNTT_OK;
    } else if (p->large.cols && batch <= p->two_pass_max) {
        // two passes per chunk of polynomials (large_chunk_bytes()).  Forward:
        // columns then rows; inverse: rows first.  Programmatic dependent
        // launches (grid_dep_start).
        const LargeInfo& li = p->large;
        if (too_large(std::max(1ull << li.L1, (1ull << li.L2) / li.cols_per_cta)))
            return fail(GBNTT_ERR_ARG, "batch too large for one launch");
        const long long n = (long long)p->hp.n;
        long long chunk = large_chunk_bytes() / (n * 4);
        if (chunk < 1) chunk = 1;
        const bool inverse = (p->hp.kind == K_R2_I32_INV);
        for (long long p0 = 0; p0 < (long long)batch; p0 += chunk) {
            const long long np = std::min<long long>(chunk, (long long)batch - p0);
            KArgs first = a, last = a;
            first.in = static_cast<const int*>(d_in) + p0 * n;
            first.out = static_cast<int*>(d_out) + p0 * n;
            first.batch = np;
            first.canonical = 0;    // the epilogue belongs to the last pass only
            first.scale = 0;
            last.in = first.out;
            last.out = first.out;
            last.batch = np;
            int L1 = li.L1, L2 = li.L2;
            void* cargs_first[] = {&first, &L2};
            void* rargs_first[] = {&first, &L1};
            void* cargs_last[] = {&last, &L2};
            void* rargs_last[] = {&last, &L1};
            const unsigned cgrid = (unsigned)(np * ((1LL << li.L2) / li.cols_per_cta));
            const unsigned rgrid = (unsigned)(((np << li.L1) + li.rows_per_cta - 1) / li.rows_per_cta);
            auto cols = [&](void** args) {
                return launch_kernel(li.cols, cgrid, li.cols_threads, li.cols_smem, args, s, true, SMEM_SHARE);
            };
            auto rows = [&](void** args) {
                return launch_kernel(li.rows, rgrid, li.rows_threads, li.rows_smem, args, s, true, SMEM_SHARE);
            };
            if (!inverse) {
                e = cols(cargs_first);
                if (e == cudaSuccess) e = rows(rargs_last);
            } else {
                e = rows(rargs_first);
                if (e == cudaSuccess) e = cols(cargs_last);
            }
            if (e != cudaSuccess) return cuda_fail(e, "kernel launch");
            g_launches.fetch_add(2, std::memory_order_relaxed);
        }
        return GBNTT_OK;
    } else if (p->fam >= 0) {
        // A launch of at most one CTA per SM is latency-bound: it takes the
        // latency form (one polynomial per CTA over up to 256 threads) where
        // the design has one, and its CTAs pull the table into L1 up front (a
        // large launch finds it there already, and the extra prefetches
        // measured 6-8 % slower for int32 and radix-8).
        const int sms = sm_count();
        const bool small = batch <= (uint64_t)sms;
        const KernelInfo& k = small && p->kl.fn ? p->kl : p->ki;
        if (batch > 0x7FFFFFFFull * (unsigned)k.polys) return fail(GBNTT_ERR_ARG, "batch too large for one launch");
        const unsigned long long blocks = (batch + k.polys - 1) / k.polys;
        // The tensor-core form from more than two tiles (of 1024 coefficients) per
        // SM: a warp takes a whole tile, so with fewer the window kernel spreads
        // over more threads.  n = 32, where two thirds of the matrix products are
        // with zeros, stays with the window kernel.  Forward + inverse after an L2
        // flush, us, window / tensor cores: 1024 x 1 8.9 / 10.9, x 152 9.4 / 10.9,
        // x 304 10.9 / 10.9, x 608 12.3 / 12.3, x 4864 25.2 / 22.0; 256 x 8 9.2 /
        // 10.3, x 1216 10.1 / 10.9, x 4864 11.8 / 10.9, x 19456 21.1 / 20.6;
        // 32 x 155648 18.6 / 20.8.
        const unsigned long long tiles = ((batch << p->hp.L) + TC_TILE - 1) / TC_TILE;
        if (p->tc_fn && tiles > 2ull * (unsigned)sms) {
            // a warp per tile; one-warp CTAs, which spread over the SMs, up to
            // the resident count
            const unsigned long long cap = (unsigned long long)TC_OCC * (unsigned)sms;
            const int threads = tiles <= cap ? 32 : TC_CTA;
            const unsigned grid = (unsigned)std::min(cap, (tiles * 32 + threads - 1) / threads);
            int L = p->hp.L;
            void* targs[] = {&a, &L};
            e = launch_kernel(p->tc_fn, grid, threads, threads / 32 * TC_WARP_RING, targs, s, true);
            if (e != cudaSuccess) return cuda_fail(e, "kernel launch");
            g_launches.fetch_add(1, std::memory_order_relaxed);
            return GBNTT_OK;
        }
        a.tab_bytes = blocks <= (unsigned long long)sms ? (int)p->tile_tab_bytes : 0;
        void* args[] = {&a};
        e = launch_kernel(k.fn, (unsigned)blocks, k.threads, k.smem, args, s, true);
    } else if (p->hp.kind == K_R8_I16_STAGE) {
        e = launch_r8_stage(a, p->hp.L, s);
    } else if (p->hp.kind == K_BITREV_I16) {
        e = launch_bitrev(a, p->hp.L, s);
    } else if (p->hp.kind == K_FULL_BARRETT_I16) {
        e = launch_full_barrett(a, (long long)batch * p->hp.n, p->hp.fb_fs, p->hp.fb_wq, s);
    }
    if (e != cudaSuccess) return cuda_fail(e, "kernel launch");
    g_launches.fetch_add(1, std::memory_order_relaxed);
    return GBNTT_OK;
}

}  // namespace

int gbntt_internal_fail(int code, const std::string& msg) { return fail(code, msg); }

void gbntt_internal_count_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }

int gbntt_internal_plan_L(const gbntt_plan* p) { return p ? p->hp.L : 0; }

void gbntt_internal_plan_args(const gbntt_plan* p, int* fam, int* L, int* elem_bytes, KArgs* a) {
    *fam = p->br ? -1 : p->fam;
    *L = p->hp.L;
    *elem_bytes = p->hp.elem_bytes;
    *a = p->base;
}

const void* gbntt_internal_mapped(const void* h) {
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, h) != cudaSuccess) {
        cudaGetLastError();   // an unknown pointer is an answer, not an error
        return nullptr;
    }
    return at.type == cudaMemoryTypeHost ? at.devicePointer : nullptr;
}

extern "C" {

int gbntt_abi_version(void) { return GBNTT_ABI_VERSION; }

const char* gbntt_last_error(void) { return g_err.c_str(); }

uint64_t gbntt_launch_count(void) { return g_launches.load(); }

const char* gbntt_status_string(int status) {
    switch (status) {
    case GBNTT_OK: return "ok";
    case GBNTT_ERR_ARG: return "invalid argument";
    case GBNTT_ERR_LENGTH: return "unsupported length";
    case GBNTT_ERR_MODULUS: return "invalid modulus";
    case GBNTT_ERR_ROOT: return "root of unity has the wrong order";
    case GBNTT_ERR_LAYERS: return "radix-4 needs an even number of layers";
    case GBNTT_ERR_KIND: return "unknown design kind";
    case GBNTT_ERR_CUDA: return "CUDA error";
    case GBNTT_ERR_NOMEM: return "out of memory";
    case GBNTT_ERR_TIMEOUT: return "timeout";
    case GBNTT_ERR_ADMISSION: return "admission refused";
    default: return "unknown status";
    }
}

int gbntt_host_tables(int kind, uint32_t n, int64_t q, int64_t root, int64_t factor, uint32_t flags,
                      int which, int64_t* dst, int64_t cap, int64_t* len) {
    HostPlan hp;
    std::string err;
    const int rc = build_host_plan(kind, n, q, root, factor, flags, hp, err);
    if (rc != GBNTT_OK) return fail(rc, err);
    std::vector<int64_t> v;
    if (which == 0) {
        v.assign(hp.tab.begin(), hp.tab.end());
    } else if (which == 1) {
        v = {hp.c, hp.r4_fneg, hp.r4_wc, hp.fb_fs, hp.fb_wq, hp.tail_wq, hp.tail_bits, hp.r8_sym, hp.stages};
    } else if (which == 2) {
        v.assign(hp.f8, hp.f8 + 64);
    } else {
        return fail(GBNTT_ERR_ARG, "unknown table selector");
    }
    if (len) *len = (int64_t)v.size();
    if (dst)
        for (int64_t i = 0; i < (int64_t)v.size() && i < cap; ++i) dst[i] = v[i];
    return GBNTT_OK;
}

int gbntt_plan_create(gbntt_plan** out, int kind, uint32_t n, int64_t q, int64_t root, int64_t factor,
                      uint32_t flags) {
    if (!out) return fail(GBNTT_ERR_ARG, "plan pointer is null");
    *out = nullptr;
    gbntt_plan* p = new (std::nothrow) gbntt_plan();
    if (!p) return fail(GBNTT_ERR_NOMEM, "host allocation failed");
    std::string err;
    int rc = build_host_plan(kind, n, q, root, factor, flags, p->hp, err);
    if (rc != GBNTT_OK) {
        delete p;
        return fail(rc, err);
    }
    const HostPlan& hp = p->hp;
    // GBNTT_FLAG_CANONICAL without GBNTT_FLAG_LANE_EXACT: the canonical family
    // of the design's direction and storage type (the two-pass int32 lengths
    // keep the reference's lane arithmetic plus the final reduction)
    const bool canon = canonical_fast(kind, hp.q, flags);
    p->fam = canon ? canonical_family(kind) : family_of(kind);
    p->br = !canon && (kind == K_R4_I16_INV);
    if (p->fam >= 0 && hp.elem_bytes == 4 && !(flags & FLAG_NATURAL_ORDER))   // two passes have no natural-order form
        p->two_pass_max = two_pass_limit(hp.L, canon, kind == K_R2_I32_INV);
    bool found = true;
    if (p->two_pass_max) {
        if (canon) p->clarge = canon_large_info(p->fam, hp.L);
        else p->large = large_info(p->fam, hp.L);
        found = canon ? p->clarge.cols != nullptr : p->large.cols != nullptr;
    }
    const int form = p->fam == F_R2F16 || p->fam == F_R2I16 ? r2_form(hp.q, hp.c) : R2_WIDE;
    if (p->fam >= 0 && p->two_pass_max != UINT64_MAX) {
        p->ki = kernel_for(p->fam, hp.L, p->br, false, form);
        p->kl = kernel_for(p->fam, hp.L, p->br, true, form);
        found = found && p->ki.fn;
    }
    if (!found) {
        delete p;
        return fail(GBNTT_ERR_LENGTH, "no kernel for this length");
    }
    cudaError_t e = cudaGetDevice(&p->device);
    if (e != cudaSuccess) {
        delete p;
        return cuda_fail(e, "cudaGetDevice");
    }
    if (p->fam >= 0 && p->ki.smem > 48 * 1024) {
        e = cudaFuncSetAttribute(p->ki.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, p->ki.smem);
        if (e != cudaSuccess) {
            delete p;
            return cuda_fail(e, "cudaFuncSetAttribute");
        }
    }
    if (p->clarge.cols) {
        e = raise_smem_limit(p->clarge.cols, p->clarge.cols_smem);
        if (e == cudaSuccess) e = raise_smem_limit(p->clarge.rows, p->clarge.rows_smem);
        if (e != cudaSuccess) {
            delete p;
            return cuda_fail(e, "cudaFuncSetAttribute");
        }
    }
    if (p->large.cols) {
        e = cudaFuncSetAttribute(p->large.cols, cudaFuncAttributeMaxDynamicSharedMemorySize, p->large.cols_smem);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(p->large.rows, cudaFuncAttributeMaxDynamicSharedMemorySize, p->large.rows_smem);
        if (e != cudaSuccess) {
            delete p;
            return cuda_fail(e, "cudaFuncSetAttribute");
        }
    }
    if (kind == K_BITREV_I16 && bitrev_smem_bytes(hp.L) > 48 * 1024) {
        e = raise_smem_limit(bitrev_kernel_ptr(), bitrev_smem_bytes(hp.L));
        if (e != cudaSuccess) {
            delete p;
            return cuda_fail(e, "cudaFuncSetAttribute");
        }
    }
    // radix-4 and wide radix-2 int16 designs: (tw, w') packed into one word
    // (both fit int16)
    const bool packed = form == R2_WIDE && (p->fam == F_R2F16 || p->fam == F_R2I16 || p->fam == F_R4F16);
    const bool inverse = (kind == K_R2_I16_INV || kind == K_R2_I32_INV || kind == K_R4_I16_INV);
    std::vector<int32_t> dev_tab;
    std::vector<uint32_t> tc_tab;
    uint32_t tc_ke = 0, tc_corr = 0;
    if (canon) {
        // canonical families: (w, w') pairs computed on the device: the table
        // of the whole transform where one CTA runs any of the plan's calls,
        // then the tables of the two passes
        const size_t n_tile = p->two_pass_max != UINT64_MAX ? canon_table_entries(hp.L, inverse) : 0;
        const size_t n_blocks = p->clarge.cols ? two_pass_entries(hp.L, p->clarge.row_el) : 0;
        p->tile_tab_bytes = n_tile * sizeof(int2);
        p->tab_bytes = (n_tile + n_blocks) * sizeof(int2);
        if (hp.elem_bytes == 2 && tc_supported(hp.L, hp.q)) {
            tc_build(hp.L, hp.q, hp.root, inverse, (flags & FLAG_NATURAL_ORDER) != 0, (flags & FLAG_SCALE_NINV) != 0,
                     tc_tab, &tc_ke, &tc_corr);
            p->tc_bytes = tc_tab.size() * sizeof(uint32_t);
        }
        e = cudaMalloc(&p->d_tab, p->tab_bytes + p->tc_bytes);
        if (e == cudaSuccess && n_blocks) e = cudaMalloc(&p->d_err, 256);
        if (e != cudaSuccess) {
            if (p->d_tab) cudaFree(p->d_tab);
            delete p;
            return e == cudaErrorMemoryAllocation ? fail(GBNTT_ERR_NOMEM, "device allocation failed")
                                                  : cuda_fail(e, "cudaMalloc");
        }
        const uint32_t q32 = (uint32_t)hp.q;
        if (n_tile) e = make_canon_table(p->d_tab, hp.L, q32, (uint32_t)hp.root, inverse, 0);
        if (n_blocks) {
            p->tab_blocks = p->d_tab + n_tile;
            if (e == cudaSuccess)
                e = make_two_pass_tables(p->d_tab + n_tile, hp.L, p->clarge.L2, p->clarge.row_el, q32, (uint32_t)hp.root,
                                         inverse, 0);
            if (e == cudaSuccess) e = cudaMemsetAsync(p->d_err, 0, 256, 0);
        }
        if (e == cudaSuccess && p->tc_bytes)
            e = cudaMemcpyAsync(reinterpret_cast<char*>(p->d_tab) + p->tab_bytes, tc_tab.data(), p->tc_bytes,
                                cudaMemcpyHostToDevice, 0);
        if (e == cudaSuccess) e = cudaStreamSynchronize(0);
        if (e != cudaSuccess) {
            cudaFree(p->d_tab);
            if (p->d_err) cudaFree(p->d_err);
            delete p;
            return cuda_fail(e, "canonical table");
        }
    } else if (packed) {
        dev_tab.resize(hp.tab.size() / 2);
        for (size_t i = 0; i < dev_tab.size(); ++i)
            dev_tab[i] = (int32_t)(((uint32_t)hp.tab[2 * i] & 0xFFFFu) | ((uint32_t)hp.tab[2 * i + 1] << 16));
    } else {
        dev_tab = hp.tab;
    }
    if (!dev_tab.empty()) {
        p->tab_bytes = p->tile_tab_bytes = dev_tab.size() * sizeof(int32_t);
        e = cudaMalloc(&p->d_tab, p->tab_bytes);
        if (e != cudaSuccess) {
            delete p;
            return e == cudaErrorMemoryAllocation ? fail(GBNTT_ERR_NOMEM, "device allocation failed")
                                                  : cuda_fail(e, "cudaMalloc");
        }
        e = cudaMemcpy(p->d_tab, dev_tab.data(), p->tab_bytes, cudaMemcpyHostToDevice);
        if (e != cudaSuccess) {
            cudaFree(p->d_tab);
            delete p;
            return cuda_fail(e, "cudaMemcpy (tables)");
        }
    }
    KArgs& a = p->base;
    std::memset(&a, 0, sizeof(a));
    a.tab = packed ? nullptr : p->d_tab;
    a.tab16 = packed ? reinterpret_cast<const int*>(p->d_tab) : nullptr;
    a.wq1 = (p->fam == F_R4F16 && hp.tab.size() >= 2) ? hp.tab[1] : 0;
    a.q = (int)hp.q;
    a.c = hp.c;
    a.fneg = hp.r4_fneg;
    a.wc = hp.r4_wc;
    if (p->fam == F_R2F16 || p->fam == F_R2I16) a.lean = form;
    a.canonical = (flags & FLAG_CANONICAL) ? 1 : 0;
    a.canon_c = hp.q >= 3 ? (int)((((uint64_t)1 << 32) + hp.q / 2) / hp.q) : 0;
    if (canon) {
        a.canonical = 1;
        a.c = (int)(2 * hp.q);
        a.cq = (unsigned)((((uint64_t)1) << 32) / (uint64_t)hp.q);
        if (hp.elem_bytes == 2) {
            const int64_t m = hp.q * ((32768 + hp.q - 1) / hp.q);     // a multiple of q, >= 2^15
            a.in_off = (int)(2 * m);
        } else {
            a.in_off = (int)(hp.q - ((int64_t)1 << 31) % hp.q);      // residue of -2^31, in (0, q]
        }
        const uint64_t ninv = (uint64_t)modinv((int64_t)hp.n, hp.q);
        a.ninv = (unsigned)ninv;
        a.ninv_q = (unsigned)((ninv << 32) / (uint64_t)hp.q);
        if (p->tc_bytes) {
            const bool natural = (flags & FLAG_NATURAL_ORDER) != 0;
            a.tctab = reinterpret_cast<const uint4*>(reinterpret_cast<const char*>(p->d_tab) + p->tab_bytes);
            a.tc_ke = (int)tc_ke;
            a.tc_corr = (int)tc_corr;
            if (hp.L > TC_MIN_L) p->tc_fn = tc16_kernel(hp.L, inverse && !natural, !inverse && !natural);
        }
    }
    a.natural_in = ((flags & FLAG_NATURAL_ORDER) && inverse) ? 1 : 0;
    a.natural_out = ((flags & FLAG_NATURAL_ORDER) && !inverse) ? 1 : 0;
    a.scale = (flags & FLAG_SCALE_NINV) ? 1 : 0;
    a.fb_fs = hp.fb_fs;
    a.fb_wq = hp.fb_wq;
    a.r8_sym = hp.r8_sym;
    // radix-8: the multiplier of the twiddle 1, also for the k = 0 outputs of
    // every stage (table entry 0 is that twiddle, in the plan's w' mode)
    a.tail_wq = (p->fam == F_R8F16 && hp.tab.size() >= 2) ? hp.tab[1] : hp.tail_wq;
    for (int i = 0; i < 64; ++i) a.f8[i] = hp.f8[i];
    for (int i = 0; i < 4; ++i) a.f8s[i] = hp.f8s[i];
    for (int i = 0; i < 16; ++i) a.ftail[i] = hp.ftail[i];
    *out = p;
    return GBNTT_OK;
}

int gbntt_plan_destroy(gbntt_plan* p) {
    if (!p) return GBNTT_OK;
    if (p->d_tab) cudaFree(p->d_tab);
    if (p->d_err) cudaFree(p->d_err);
    if (p->d_stage) cudaFree(p->d_stage);
    if (p->zc_state) gbntt_internal_zc_free(p->zc_state);
    delete p;
    return GBNTT_OK;
}

int gbntt_plan_status(const gbntt_plan* p) {
    if (!p) return fail(GBNTT_ERR_ARG, "plan is null");
    if (!p->d_err) return GBNTT_OK;
    unsigned w = 0;
    cudaError_t e = cudaMemcpy(&w, p->d_err, sizeof(w), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return cuda_fail(e, "status read");
    if (!w) return GBNTT_OK;
    e = cudaMemset(p->d_err, 0, sizeof(w));
    if (e != cudaSuccess) return cuda_fail(e, "status reset");
    return fail(GBNTT_ERR_TIMEOUT, "a tile load of the column pass did not arrive within the wait limit");
}

int gbntt_plan_query(const gbntt_plan* p, int what, int64_t* value) {
    if (!p || !value) return fail(GBNTT_ERR_ARG, "null argument");
    switch (what) {
    case GBNTT_Q_N: *value = p->hp.n; break;
    case GBNTT_Q_MODULUS: *value = p->hp.q; break;
    case GBNTT_Q_ELEM_BYTES: *value = p->hp.elem_bytes; break;
    case GBNTT_Q_STAGES: *value = p->hp.stages; break;
    case GBNTT_Q_KIND: *value = p->hp.kind; break;
    case GBNTT_Q_TABLE_BYTES: *value = (int64_t)(p->tab_bytes + p->tc_bytes); break;
    default: return fail(GBNTT_ERR_ARG, "unknown query");
    }
    return GBNTT_OK;
}

int gbntt_execute(const gbntt_plan* p, const void* d_in, void* d_out, uint64_t batch, void* stream) {
    if (!p) return fail(GBNTT_ERR_ARG, "plan is null");
    if (batch == 0) return GBNTT_OK;
    if (!d_in || !d_out) return fail(GBNTT_ERR_ARG, "null buffer");
    if ((reinterpret_cast<uintptr_t>(d_in) | reinterpret_cast<uintptr_t>(d_out)) & 15)
        return fail(GBNTT_ERR_ARG, "device buffers must be 16-byte aligned");
    if (p->hp.kind == K_R8_I16_STAGE && d_in == d_out)
        return fail(GBNTT_ERR_ARG, "the radix-8 stage cannot run in place");
    return launch(p, d_in, d_out, batch, static_cast<cudaStream_t>(stream));
}

int gbntt_execute_host(gbntt_plan* p, const void* h_in, void* h_out, uint64_t batch, void* stream) {
    if (!p) return fail(GBNTT_ERR_ARG, "plan is null");
    if (batch == 0) return GBNTT_OK;
    if (!h_in || !h_out) return fail(GBNTT_ERR_ARG, "null buffer");
    std::lock_guard<std::mutex> lock(p->stage_mu);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    {
        // page-locked, mapped host buffers: the zero-copy persistent kernel reads
        // and writes them directly, both directions of the link at once
        const void* mi = gbntt_internal_mapped(h_in);
        const void* mo = gbntt_internal_mapped(h_out);
        if (mi && mo && !((reinterpret_cast<uintptr_t>(mi) | reinterpret_cast<uintptr_t>(mo)) & 15) &&
            !(p->hp.kind == K_R8_I16_STAGE && h_in == h_out)) {
            const int rc = gbntt_internal_zc_plan(&p->zc_state, p, mi, const_cast<void*>(mo), batch, s);
            if (rc == GBNTT_OK) {
                const cudaError_t e = cudaStreamSynchronize(s);
                return e == cudaSuccess ? GBNTT_OK : cuda_fail(e, "cudaStreamSynchronize");
            }
            if (rc != GBNTT_ERR_KIND) return rc;
        }
    }
    const size_t bytes = (size_t)batch * p->hp.n * (size_t)p->hp.elem_bytes;
    // the radix-8 stage reads other threads' outputs, so it gets its own output half
    const bool split = (p->hp.kind == K_R8_I16_STAGE);
    const size_t need = split ? 2 * bytes : bytes;
    cudaError_t e;
    if (p->stage_bytes < need) {
        if (p->d_stage) cudaFree(p->d_stage);
        p->d_stage = nullptr;
        p->stage_bytes = 0;
        e = cudaMalloc(&p->d_stage, need);
        if (e != cudaSuccess) return fail(GBNTT_ERR_NOMEM, "staging allocation failed");
        p->stage_bytes = need;
    }
    void* d_out = split ? static_cast<char*>(p->d_stage) + bytes : p->d_stage;
    e = cudaMemcpyAsync(p->d_stage, h_in, bytes, cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) return cuda_fail(e, "cudaMemcpyAsync H2D");
    int rc = launch(p, p->d_stage, d_out, batch, s);
    if (rc != GBNTT_OK) return rc;
    e = cudaMemcpyAsync(h_out, d_out, bytes, cudaMemcpyDeviceToHost, s);
    if (e != cudaSuccess) return cuda_fail(e, "cudaMemcpyAsync D2H");
    e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_fail(e, "cudaStreamSynchronize");
    return GBNTT_OK;
}

}  // extern "C"
