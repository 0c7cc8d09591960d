// C ABI of spinsim_b200 (declared in include/spinsim_b200.h): plans, launches, user-field linking.
//
// Built-in field kernels are compiled into this library as sm_100a SASS.  Kernels for user fields
// are embedded as LTO-IR (one fatbin per method variant) and linked at plan creation with the
// user's LTO-IR through nvJitLink (loaded with dlopen from the CUDA toolkit), then loaded with the
// runtime's library API.
#include <cuda_runtime.h>
#include <dlfcn.h>
#include <math.h>
#include <stdarg.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <list>
#include <mutex>
#include <new>
#include <string>
#include <vector>

#include "../../include/spinsim_b200.h"
#include "common.cuh"
#define SPINSIM_SCAN_KERNELS 1
#include "scan.cuh"

using namespace spinsim;

// ------------------------------------------------------------------ layout checks
static_assert(sizeof(spinsim_table) == sizeof(TableChannel), "table layout");
static_assert(sizeof(spinsim_field) == sizeof(FieldDesc), "field layout");
static_assert(sizeof(spinsim_instance) == sizeof(Instance), "instance layout");
static_assert(offsetof(spinsim_instance, psi0) == offsetof(Instance, psi0), "instance psi0");
static_assert(SPINSIM_MAX_CALL_PARAMS == kSingleParams, "parameters by value");
static_assert(offsetof(spinsim_field, bias) == offsetof(FieldDesc, bias), "field bias");

// ------------------------------------------------------------------ errors
static thread_local std::string g_error;

static int fail(int code, const char* fmt, ...) {
    char buf[1024];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    g_error = buf;
    return code;
}

#define CUDA_TRY(expr)                                                                          \
    do {                                                                                        \
        cudaError_t e_ = (expr);                                                                \
        if (e_ != cudaSuccess)                                                                  \
            return fail(SPINSIM_ERR_CUDA, "%s failed: %s (%s:%d)", #expr, cudaGetErrorString(e_), \
                        __FILE__, __LINE__);                                                    \
    } while (0)

// ------------------------------------------------------------------ kernel registry
typedef const void* (*kernel_getter)(void);
struct BuiltinEntry {
    int dims, integ, expo_h, expo_o, field, prec, minb;
    kernel_getter get;
};
struct UserEntry {
    int dims, integ, expo_h, expo_o, prec, minb;
    const unsigned char* begin;
    const unsigned char* end;
};
struct DmmaEntry {
    int dims, prec, minb;
    kernel_getter get;
};
// Generated by the build: declares the getters/blobs and defines kBuiltin[], kUser[].
#include "registry_gen.inc"

// ------------------------------------------------------------------ nvJitLink (dlopen)
namespace {
typedef int (*jl_create_t)(void** handle, uint32_t n, const char** opts);
typedef int (*jl_add_t)(void* handle, int type, const void* data, size_t size, const char* name);
typedef int (*jl_complete_t)(void* handle);
typedef int (*jl_size_t)(void* handle, size_t* size);
typedef int (*jl_get_t)(void* handle, void* out);
typedef int (*jl_log_t)(void* handle, char* out);
typedef int (*jl_destroy_t)(void** handle);

struct JitLink {
    void* so = nullptr;
    jl_create_t create;
    jl_add_t add;
    jl_complete_t complete;
    jl_size_t cubin_size;
    jl_get_t cubin;
    jl_size_t log_size;
    jl_log_t log;
    jl_destroy_t destroy;
};
std::mutex g_jl_mutex;
JitLink g_jl;

int load_jitlink() {
    std::lock_guard<std::mutex> lock(g_jl_mutex);
    if (g_jl.so) return SPINSIM_OK;
    const char* candidates[] = {getenv("SPINSIM_NVJITLINK"), "/usr/local/cuda/lib64/libnvJitLink.so.12",
                                "/usr/local/cuda/lib64/libnvJitLink.so", "libnvJitLink.so.12"};
    void* so = nullptr;
    for (const char* c : candidates) {
        if (!c) continue;
        so = dlopen(c, RTLD_NOW | RTLD_LOCAL);
        if (so) break;
    }
    if (!so) return fail(SPINSIM_ERR_LINK, "cannot load libnvJitLink: %s", dlerror());
    // The 12.x entry points are versioned; use the oldest name that has every call used here.
    g_jl.create = (jl_create_t)dlsym(so, "__nvJitLinkCreate_12_0");
    g_jl.add = (jl_add_t)dlsym(so, "__nvJitLinkAddData_12_0");
    g_jl.complete = (jl_complete_t)dlsym(so, "__nvJitLinkComplete_12_0");
    g_jl.cubin_size = (jl_size_t)dlsym(so, "__nvJitLinkGetLinkedCubinSize_12_0");
    g_jl.cubin = (jl_get_t)dlsym(so, "__nvJitLinkGetLinkedCubin_12_0");
    g_jl.log_size = (jl_size_t)dlsym(so, "__nvJitLinkGetErrorLogSize_12_0");
    g_jl.log = (jl_log_t)dlsym(so, "__nvJitLinkGetErrorLog_12_0");
    g_jl.destroy = (jl_destroy_t)dlsym(so, "__nvJitLinkDestroy_12_0");
    if (!g_jl.create || !g_jl.add || !g_jl.complete || !g_jl.cubin_size || !g_jl.cubin || !g_jl.log_size ||
        !g_jl.log || !g_jl.destroy) {
        dlclose(so);
        return fail(SPINSIM_ERR_LINK, "libnvJitLink lacks the 12.0 entry points");
    }
    g_jl.so = so;
    return SPINSIM_OK;
}

enum { JL_INPUT_LTOIR = 3, JL_INPUT_FATBIN = 4 };

int jit_link(const void* kernel_fatbin, size_t kernel_size, const void* user_ltoir, size_t user_size,
             std::vector<char>* cubin) {
    int rc = load_jitlink();
    if (rc) return rc;
    std::vector<std::string> opts = {"-arch=sm_100a", "-lto", "-O3"};
    std::vector<const char*> optp;
    for (auto& s : opts) optp.push_back(s.c_str());
    void* h = nullptr;
    if (g_jl.create(&h, (uint32_t)optp.size(), optp.data()) != 0) return fail(SPINSIM_ERR_LINK, "nvJitLinkCreate failed");
    auto log_fail = [&](const char* what) {
        size_t n = 0;
        std::string log;
        if (g_jl.log_size(h, &n) == 0 && n > 1) {
            log.resize(n);
            g_jl.log(h, &log[0]);
        }
        g_jl.destroy(&h);
        return fail(SPINSIM_ERR_LINK, "%s: %s", what, log.c_str());
    };
    if (g_jl.add(h, JL_INPUT_FATBIN, kernel_fatbin, kernel_size, "spinsim_kernels") != 0)
        return log_fail("adding the kernel LTO-IR failed");
    if (g_jl.add(h, JL_INPUT_LTOIR, user_ltoir, user_size, "user_field") != 0)
        return log_fail("adding the user field LTO-IR failed");
    if (g_jl.complete(h) != 0) return log_fail("nvJitLink failed to link the user field");
    size_t n = 0;
    if (g_jl.cubin_size(h, &n) != 0 || n == 0) return log_fail("no linked cubin");
    cubin->resize(n);
    if (g_jl.cubin(h, cubin->data()) != 0) return log_fail("reading the linked cubin failed");
    g_jl.destroy(&h);
    return SPINSIM_OK;
}

// The last kernels linked, by everything that goes into a link (the built-in kernel's image and the field's whole
// LTO-IR), most recent first: another plan of the same field, which a program that makes a
// simulator per call asks for, takes a copy. Even from its disk cache nvJitLink needs milliseconds, more the
// larger the kernel's image. At most kLinkedKept entries.
struct Linked {
    const void* kernel;
    std::string field;
    std::vector<char> cubin;
};
constexpr size_t kLinkedKept = 8;
std::mutex g_linked_mutex;
std::list<Linked> g_linked;

int linked_cubin(const void* kernel_fatbin, size_t kernel_size, const void* user_ltoir, size_t user_size,
                 std::vector<char>* cubin) {
    try {
        const std::string field((const char*)user_ltoir, user_size);
        auto is_this = [&](const Linked& k) {
            return k.kernel == kernel_fatbin && k.field == field;
        };
        {
            std::lock_guard<std::mutex> lock(g_linked_mutex);
            auto at = std::find_if(g_linked.begin(), g_linked.end(), is_this);
            if (at != g_linked.end()) {
                g_linked.splice(g_linked.begin(), g_linked, at);
                *cubin = at->cubin;
                return SPINSIM_OK;
            }
        }
        const int rc = jit_link(kernel_fatbin, kernel_size, user_ltoir, user_size, cubin);
        if (rc) return rc;
        std::lock_guard<std::mutex> lock(g_linked_mutex);
        if (std::none_of(g_linked.begin(), g_linked.end(), is_this))
            g_linked.push_front(Linked{kernel_fatbin, field, *cubin});
        if (g_linked.size() > kLinkedKept) g_linked.pop_back();
        return SPINSIM_OK;
    } catch (const std::bad_alloc&) {
        return fail(SPINSIM_ERR_LINK, "out of host memory while linking the user field");
    }
}
}  // namespace

// ------------------------------------------------------------------ plan
struct spinsim_plan {
    spinsim_plan_desc desc;
    MethodConfig m;
    const void* func = nullptr;   // host stub or cudaKernel_t
    cudaLibrary_t lib = nullptr;
    int block = kEvolveThreadsDefault;
    int blocks_per_sm = 1;
    int sm_count = 148;
    int regs = 0;
    int device = 0;
    int smem_per_warp = 0;  // dynamic shared memory of the FP32-bulk tone kernels
    bool lockstep = false;  // kernel needs one lane per output interval (tone synthesis)
    int intervals_per_lane = 1;
    bool cta_tiles = false;  // a tile is a CTA's unit of work (the tensor-path tone kernel), not a warp's
    spinsim_plan* tensor = nullptr;  // FP64 Magnus CF4 tone plans: the tensor-path form, for the fields it takes
};

// Output intervals in one tile of the plan's time-evolution kernel.
static int tile_intervals(const spinsim_plan* p, int lanes) {
    return p->cta_tiles ? kDmmaTile : 32 * p->intervals_per_lane / lanes;
}

// The plan's warps (one lane per output interval) or CTAs (FP64 tensor path) take 32 consecutive output
// intervals: a tile of the state scan, whose product they write.
static bool writes_products(const spinsim_plan* p, int lanes) {
    return p->cta_tiles ? p->desc.precision == SPINSIM_PRECISION_FP64 : !p->lockstep && lanes == 1;
}

extern "C" const char* spinsim_version(void) { return "spinsim_b200 0.1.0 (sm_100a)"; }

extern "C" int spinsim_last_error(char* buf, size_t n) {
    if (buf && n) {
        strncpy(buf, g_error.c_str(), n - 1);
        buf[n - 1] = 0;
    }
    return (int)g_error.size();
}

extern "C" int spinsim_normalise_steps(double t0, double t1, double dt_int, double dt_out, double* dt_int_out,
                                       int64_t* n_out, int32_t* n_fine, int32_t* warned) {
    if (!(dt_out > 0) || !(dt_int > 0)) return fail(SPINSIM_ERR_INVALID, "time steps must be positive");
    // I:1025-1028 (Python round() is round-half-to-even; nearbyint under the default rounding mode)
    const double ratio = dt_out / dt_int;
    const double dti = dt_out / nearbyint(ratio > 1.0 ? ratio : 1.0);
    if (dt_int_out) *dt_int_out = dti;
    if (warned) *warned = fabs(ratio - nearbyint(ratio)) > 1e-6 ? 1 : 0;
    // I:1034
    const double n = (t1 - t0) / dt_out;
    if (n_out) *n_out = n > 0 ? (int64_t)n : 0;
    // I:832
    if (n_fine) *n_fine = (int32_t)floor(dt_out / dti + 0.5);
    return SPINSIM_OK;
}

static bool valid_expo(int dim, int e) {
    if (dim == 2) return e == EXPO_ANALYTIC || e == EXPO_LIE_TROTTER;
    return e == EXPO_LIE_TROTTER || e == EXPO_LIE_TROTTER_8;
}

// Make p a tensor-path tone plan (Magnus CF4).  Register budgets: 128 registers (4 CTAs per SM) by default;
// budgets of at most 85 registers take the 6-CTA build (80 registers), at most 102 the 5-CTA build (96), above
// 128 the 168-register build.
static void take_tensor_path(spinsim_plan* p) {
    const int mr = p->desc.max_registers;
    const int want_minb = (mr > 0 && mr <= 85) ? 6 : (mr > 0 && mr <= 102) ? 5 : (mr == 0 || mr <= 128) ? 4 : 3;
    p->func = nullptr;
    for (int minb = want_minb; minb >= 3 && !p->func; minb--)
        for (const DmmaEntry& k : kDmma)
            if (k.dims == p->desc.spin_dim && k.prec == p->desc.precision && k.minb == minb) {
                p->func = k.get();
                break;
            }
    p->block = kDmmaThreads;
    p->cta_tiles = true;
    p->lockstep = true;
    p->m.lanes = 1;
}

// The kernel's attributes and resident CTAs.
static cudaError_t query_kernel(spinsim_plan* p) {
    cudaFuncAttributes attr;
    cudaError_t e = cudaFuncGetAttributes(&attr, p->func);
    if (e == cudaSuccess && p->smem_per_warp) {
        e = cudaFuncSetAttribute(p->func, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 kEvolveThreadsMax / 32 * p->smem_per_warp);
        // prefer the largest shared-memory carve-out so that shared memory does not cap residency
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(p->func, cudaFuncAttributePreferredSharedMemoryCarveout,
                                     (int)cudaSharedmemCarveoutMaxShared);
    }
    if (e != cudaSuccess) return e;
    p->regs = attr.numRegs;
    if (p->block > attr.maxThreadsPerBlock) p->block = attr.maxThreadsPerBlock / 32 * 32;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&p->blocks_per_sm, p->func, p->block,
                                                      (size_t)(p->block / 32) * p->smem_per_warp);
    if (p->blocks_per_sm < 1) p->blocks_per_sm = 1;
    return e;
}

extern "C" int spinsim_plan_create(const spinsim_plan_desc* desc, const void* field_ltoir, size_t field_ltoir_size,
                                   spinsim_plan** out) {
    if (!desc || !out) return fail(SPINSIM_ERR_INVALID, "null argument");
    *out = nullptr;
    const spinsim_plan_desc& d = *desc;
    if (d.spin_dim != 0 && d.spin_dim != 2 && d.spin_dim != 3)
        return fail(SPINSIM_ERR_INVALID, "spin_dim must be 2, 3 or 0 (mixed), got %d", d.spin_dim);
    if (d.integration < 0 || d.integration > 2) return fail(SPINSIM_ERR_INVALID, "bad integration %d", d.integration);
    if (d.spin_dim != 3 && !valid_expo(2, d.expo_half))
        return fail(SPINSIM_ERR_INVALID, "exponentiation %d is not available for spin half", d.expo_half);
    if (d.spin_dim != 2 && !valid_expo(3, d.expo_one))
        return fail(SPINSIM_ERR_INVALID, "exponentiation %d is not available for spin one", d.expo_one);
    if (d.number_of_squares < 0) return fail(SPINSIM_ERR_INVALID, "number_of_squares must be >= 0");
    if (d.field_kind < 0 || d.field_kind > 2) return fail(SPINSIM_ERR_INVALID, "bad field kind %d", d.field_kind);
    if (d.precision != 0 && d.precision != 1) return fail(SPINSIM_ERR_INVALID, "bad precision %d", d.precision);
    if (d.threads_per_block && (d.threads_per_block % 32 || d.threads_per_block > kEvolveThreadsMax || d.threads_per_block < 32))
        return fail(SPINSIM_ERR_INVALID, "threads_per_block must be a multiple of 32 in [32, %d]", kEvolveThreadsMax);
    if (d.lanes && (d.lanes & (d.lanes - 1) || d.lanes > 32)) return fail(SPINSIM_ERR_INVALID, "lanes must be a power of two <= 32");
    if (d.variant < 0 || d.variant > 1) return fail(SPINSIM_ERR_INVALID, "bad kernel variant %d", d.variant);
    if ((d.field_kind == SPINSIM_FIELD_USER) != (field_ltoir != nullptr))
        return fail(SPINSIM_ERR_INVALID, "field_ltoir is required for user fields and only for them");

    // Canonical variant key: unused exponentiators are fixed so a single-dimension plan matches.
    const int eh = d.spin_dim == 3 ? EXPO_ANALYTIC : d.expo_half;
    const int eo = d.spin_dim == 2 ? EXPO_LIE_TROTTER : d.expo_one;

    spinsim_plan* p = new spinsim_plan();
    p->desc = d;
    int h = (d.number_of_squares + 1) / 2;  // ceil(n / 2), I:1547
    if (h < 0) h = 0;
    p->m.integration = d.integration;
    p->m.expo_half = eh;
    p->m.expo_one = eo;
    p->m.rotating = d.rotating ? 1 : 0;
    p->m.hypercubes = h;
    p->m.precision = ldexp(1.0, 2 * h);  // 4 ** h, I:1550
    // The symmetric splitting of N = 4^h factors differs from the exponential by less than
    // |g|^3 / (8 N^2); at |g|^3 <= 2^-53 N^2 that is an eighth of a rounding error.
    p->m.lt_norm2_max = pow(ldexp(1.0, 4 * h - 53), 2.0 / 3.0);
    p->m.lanes = d.lanes;
    if (d.threads_per_block) p->block = d.threads_per_block;

    cudaError_t e = cudaGetDevice(&p->device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&p->sm_count, cudaDevAttrMultiProcessorCount, p->device);
    if (e != cudaSuccess) {
        delete p;
        return fail(SPINSIM_ERR_CUDA, "no CUDA device: %s", cudaGetErrorString(e));
    }

    const bool dmma = d.field_kind == SPINSIM_FIELD_TONES && d.precision == SPINSIM_PRECISION_FP32_BULK &&
                      d.integration == SPINSIM_INTEGRATION_MAGNUS_CF4 && d.variant == SPINSIM_VARIANT_TENSOR;
    if (dmma) {
        take_tensor_path(p);
    } else if (d.field_kind != SPINSIM_FIELD_USER) {
        // Register budget: the kernel built for MINB resident 128-thread CTAs per SM whose cap is the
        // largest that fits max_registers: 6 -> 80, 5 -> 96, 4 -> 128, 3 -> 168 registers, 2 uncapped.
        // Budgets of 80 and 96 exist only for some kernels; without one the next larger budget is taken.
        // By default 128, except for the eight-generator exponential, whose 3 x 3 temporaries would
        // spill: a launch of 400 pulse trains (FP32-bulk tables) takes 677 us at 168, 564 at 128, 561 at 96
        // and 519 at 80, where an interpolated table's steps spill too much.
        const int mr = d.max_registers;
        const int want_minb = mr <= 0 ? (eo == EXPO_LIE_TROTTER_8 ? 2 : 4) : mr <= 80 ? 6 : mr <= 96 ? 5 : mr <= 128 ? 4 : mr <= 168 ? 3 : 2;
        for (int minb = want_minb; minb >= 2 && !p->func; minb--) {
            for (const BuiltinEntry& b : kBuiltin) {
                if (b.dims == d.spin_dim && b.integ == d.integration && b.expo_h == eh && b.expo_o == eo &&
                    b.field == d.field_kind && b.prec == d.precision && b.minb == minb) {
                    p->func = b.get();
                    break;
                }
            }
        }
    } else {
        // The default image's registers are capped (96 for spin half, 128 with spin one), which a field of many live
        // values outgrows.  Fields of 25 / 49 / 81 live doubles, 2048 instances of 200 x 50 steps, spin half: 1157 / 1721 /
        // 3881 us there, 1087 / 1689 / 2496 in the uncapped image (the last in the table); spin one 1163 / 1766 / 2631 and
        // 1144 / 1722 / 2519.  A budget above 168 takes the uncapped one, and so does, without a budget, a spin-half
        // field that makes the default one spill (300 to 376 bytes of local memory, 40 to 72 without).
        const UserEntry *capped = nullptr, *uncapped = nullptr;
        for (const UserEntry& x : kUser)
            if (x.dims == d.spin_dim && x.integ == d.integration && x.expo_h == eh && x.expo_o == eo && x.prec == d.precision) {
                if (!capped) capped = &x;
                uncapped = &x;
            }
        auto load = [&](const UserEntry* u) -> int {
            if (p->lib) cudaLibraryUnload(p->lib);
            p->lib = nullptr;
            std::vector<char> cubin;
            int rc = linked_cubin(u->begin, (size_t)(u->end - u->begin), field_ltoir, field_ltoir_size, &cubin);
            if (rc) return rc;
            e = cudaLibraryLoadData(&p->lib, cubin.data(), nullptr, nullptr, 0, nullptr, nullptr, 0);
            cudaKernel_t k = nullptr;
            if (e == cudaSuccess) e = cudaLibraryGetKernel(&k, p->lib, "spinsim_evolve_user");
            if (e != cudaSuccess) return fail(SPINSIM_ERR_LINK, "loading the linked module failed: %s", cudaGetErrorString(e));
            p->func = (const void*)k;
            return SPINSIM_OK;
        };
        if (capped) {
            int rc = load(d.max_registers > 168 ? uncapped : capped);
            cudaFuncAttributes attr;
            if (!rc && d.max_registers <= 0 && d.spin_dim == 2 && cudaFuncGetAttributes(&attr, p->func) == cudaSuccess &&
                attr.localSizeBytes > 200)
                rc = load(uncapped);
            if (rc) {
                if (p->lib) cudaLibraryUnload(p->lib);
                delete p;
                return rc;
            }
        }
    }
    if (!p->func) {
        delete p;
        return fail(SPINSIM_ERR_UNSUPPORTED,
                    "no kernel built for spin_dim=%d integration=%d expo=(%d,%d) field=%d precision=%d", d.spin_dim,
                    d.integration, eh, eo, d.field_kind, d.precision);
    }
    if (d.field_kind == SPINSIM_FIELD_TONES && d.precision == SPINSIM_PRECISION_FP32_BULK && !dmma &&
        d.integration == SPINSIM_INTEGRATION_MAGNUS_CF4) {  // the warp tone synthesis
        p->smem_per_warp = kToneSharedBytes;
        p->lockstep = true;
        p->intervals_per_lane = kSynthIntervals;
        p->m.lanes = 1;
    }
    e = query_kernel(p);
    if (e == cudaSuccess && d.field_kind == SPINSIM_FIELD_TONES && d.precision == SPINSIM_PRECISION_FP64 &&
        d.integration == SPINSIM_INTEGRATION_MAGNUS_CF4 && eo != EXPO_LIE_TROTTER_8) {
        p->tensor = new spinsim_plan(*p);
        take_tensor_path(p->tensor);
        e = query_kernel(p->tensor);
    }
    if (e != cudaSuccess) {
        if (p->lib) cudaLibraryUnload(p->lib);
        delete p->tensor;
        delete p;
        return fail(SPINSIM_ERR_CUDA, "querying the kernel failed: %s", cudaGetErrorString(e));
    }
    *out = p;
    return SPINSIM_OK;
}

extern "C" int spinsim_plan_destroy(spinsim_plan* plan) {
    if (!plan) return SPINSIM_OK;
    if (plan->lib) cudaLibraryUnload(plan->lib);
    delete plan->tensor;
    delete plan;
    return SPINSIM_OK;
}

extern "C" int spinsim_plan_get_info(const spinsim_plan* plan, spinsim_plan_info* info) {
    if (!plan || !info) return fail(SPINSIM_ERR_INVALID, "null argument");
    if (plan->tensor) plan = plan->tensor;  // the kernel of nearly every tone field
    info->registers_per_thread = plan->regs;
    info->threads_per_block = plan->block;
    info->blocks_per_sm = plan->blocks_per_sm;
    info->sm_count = plan->sm_count;
    info->lanes = plan->m.lanes;
    info->linked = plan->lib != nullptr;
    const bool bulk_tones = plan->desc.field_kind == SPINSIM_FIELD_TONES &&
                            plan->desc.precision == SPINSIM_PRECISION_FP32_BULK &&
                            plan->desc.integration == SPINSIM_INTEGRATION_MAGNUS_CF4;
    info->variant = !bulk_tones ? -1 : plan->cta_tiles ? SPINSIM_VARIANT_TENSOR : SPINSIM_VARIANT_SYNTH;
    info->tile_intervals = tile_intervals(plan, plan->m.lanes ? plan->m.lanes : 1);
    return SPINSIM_OK;
}

// ------------------------------------------------------------------ workspace carving
namespace {
struct Carver {
    char* base;
    size_t used = 0;
    explicit Carver(void* b) : base((char*)b) {}
    template <class T>
    T* take(size_t count) {
        used = (used + 255) & ~(size_t)255;
        T* r = base ? (T*)(base + used) : nullptr;
        used += count * sizeof(T);
        return r;
    }
};

// Lanes per output interval.  A lane's chain is its start-up (frame sample and phasors), its share of the
// fine steps and one product per level of the lanes' combination; the launch takes that chain's latency
// while the FP64 pipes have room (up to about two warps per scheduler at a chain's own parallelism) and
// its throughput beyond.  The lane count with the least of that is taken, in units of FP64 operations.
// Measured (whole calls): 4001 x 50 steps with a quadratic shift 36 / 33 / 39 / 48 us at 4 / 8 / 16 / 32 lanes,
// 5003 x 37 of a cubic waveform 49 / 33 / 40 / 44, 100,000 x 10 of a drive 59 / 64 us at 1 / 2.
int pick_lanes(const spinsim_plan* p, int64_t intervals, int max_fine) {
    if (p->lockstep) return 1;
    if (p->m.lanes) return p->m.lanes;
    const double start = 300.0, step = 200.0, level = 60.0, saturated = 2.0;
    double best = 0.0;
    int lanes = 1;
    for (int l = 1, levels = 0; l <= 32 && l <= std::max(1, max_fine); l *= 2, levels++) {
        const double warps = (double)intervals * l / (32.0 * 4.0 * p->sm_count);  // per scheduler
        const double chain = start + step * ((max_fine + l - 1) / l) + level * levels;
        const double cost = chain * std::max(saturated, warps);
        if (l == 1 || cost < best) {
            best = cost;
            lanes = l;
        }
    }
    return lanes;
}

// Scan tiles of kScanTile output steps, every instance's in order (spin-half instances first, then
// spin one, each run padded with empty tiles to whole warps so that a warp's tiles share a
// dimension); begin/end index them per instance.
// The scan's tiles: every spin-half instance's 32-step tiles, padded to whole warps, then every
// spin-one instance's.  count_scan_plan gives the sizes, fill_scan_plan writes the tiles and each
// instance's [begin, end) range (into the staging image of the descriptors, or host vectors).
struct ScanPlan {
    int64_t n_tiles = 0;
    int64_t tiles_half = 0;  // tiles [0, tiles_half) are spin half, the rest spin one
    int64_t max_tiles = 0;   // of the longest instance
    int32_t n_instances = 0;
};

void count_scan_plan(const Instance* inst, int n_inst, ScanPlan* sp) {
    int64_t count = 0;
    for (int dim = 2; dim <= 3; dim++) {
        for (int i = 0; i < n_inst; i++)
            if (inst[i].dim == dim) {
                const int64_t tiles = (inst[i].n_out + kScanTile - 1) / kScanTile;
                count += tiles;
                sp->max_tiles = std::max(sp->max_tiles, tiles);
            }
        count = (count + kScanTilesPerWarp - 1) / kScanTilesPerWarp * kScanTilesPerWarp;
        if (dim == 2) sp->tiles_half = count;
    }
    sp->n_tiles = count;
    sp->n_instances = n_inst;
}

void fill_scan_plan(const Instance* inst, int n_inst, Tile* tiles, int32_t* begin, int32_t* end) {
    int64_t at = 0;
    for (int dim = 2; dim <= 3; dim++) {
        for (int i = 0; i < n_inst; i++) {
            if (inst[i].dim != dim) continue;
            begin[i] = (int32_t)at;
            for (int64_t f = 0; f < inst[i].n_out; f += kScanTile) {
                Tile& t = tiles[at++];
                t.instance = i;
                t.first = f;
                t.count = (int32_t)std::min<int64_t>(kScanTile, inst[i].n_out - f);
            }
            end[i] = (int32_t)at;
        }
        while (at % kScanTilesPerWarp) tiles[at++] = Tile{0, 0, 0};
    }
}

int64_t scan_tiles_of(int64_t n_out) { return (n_out + kScanTile - 1) / kScanTile; }

struct ScanBuffers {
    Tile* tiles;  // null: one instance, implicit tiles
    int32_t *begin, *end;
    double *tile_product, *tile_prefix;
    int64_t n_tiles;
    int64_t tiles_half;  // tiles [0, tiles_half) are spin half, the rest spin one
    int64_t max_tiles;   // of the longest instance
    int32_t n_instances;
};

// The descriptors (tiles, per-instance ranges) and the scratch (tile products and prefixes) are
// carved separately so a batch can keep all its descriptors in one leading block of the workspace.
void carve_scan_desc(Carver& c, const ScanPlan& sp, ScanBuffers* b) {
    b->n_tiles = sp.n_tiles;
    b->tiles_half = sp.tiles_half;
    b->max_tiles = sp.max_tiles;
    b->n_instances = sp.n_instances;
    b->tiles = c.take<Tile>((size_t)std::max<int64_t>(1, sp.n_tiles));
    b->begin = c.take<int32_t>((size_t)std::max<int32_t>(1, sp.n_instances));
    b->end = c.take<int32_t>((size_t)std::max<int32_t>(1, sp.n_instances));
}

void carve_scan_scratch(Carver& c, int64_t n_tiles, ScanBuffers* b) {
    b->tile_product = c.take<double>((size_t)std::max<int64_t>(1, n_tiles) * kScanMat);
    b->tile_prefix = c.take<double>((size_t)std::max<int64_t>(1, n_tiles) * kScanMat);
}

// One instance: implicit tiles, nothing to upload; only the scratch is carved.
void carve_scan_single(Carver& c, int64_t n_out, int32_t dim, ScanBuffers* b) {
    b->tiles = nullptr;
    b->begin = b->end = nullptr;
    b->n_tiles = scan_tiles_of(n_out);
    b->tiles_half = dim == 2 ? b->n_tiles : 0;
    b->max_tiles = b->n_tiles;
    b->n_instances = 1;
    carve_scan_scratch(c, b->n_tiles, b);
}

int upload(void* dst, const void* src, size_t bytes, cudaStream_t s) {
    if (!bytes) return SPINSIM_OK;
    CUDA_TRY(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s));
    return SPINSIM_OK;
}

enum ScanStages { SCAN_PREFIX = 1, SCAN_APPLY = 2, SCAN_ALL = 3 };

// A kernel launch (of clusters of `cluster` CTAs) that may start before the preceding kernel in the stream has completed
// (programmatic stream serialization): the kernel itself waits for that kernel's results
// (grid_dependency_wait) where it first needs them.
template <typename... K, typename... A>
cudaError_t launch_early_cluster(void (*kernel)(K...), unsigned cluster, dim3 grid, dim3 block, size_t smem,
                                 cudaStream_t s, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = cluster;
    at[1].val.clusterDim.y = 1;
    at[1].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

template <typename... K, typename... A>
cudaError_t launch_early(void (*kernel)(K...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A... args) {
    return launch_early_cluster(kernel, 1, grid, block, smem, s, args...);
}

// Multiprocessors of the current device (looked up once per device; not a stream operation).
int device_sm_count(int* out) {
    static std::mutex mu;
    static std::vector<int> known;
    int dev = 0;
    CUDA_TRY(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> g(mu);
    if (dev >= (int)known.size()) known.resize(dev + 1, 0);
    if (!known[dev]) CUDA_TRY(cudaDeviceGetAttribute(&known[dev], cudaDevAttrMultiProcessorCount, dev));
    *out = known[dev];
    return SPINSIM_OK;
}

// Output steps of a single instance up to which the whole scan is one launch of one cluster: one step per
// thread to 2048, up to kClusterSteps beyond.  Measured against the three launches (spin half / one): 100
// steps 9.4 / 16.7 -> 3.1 / 5.7 us, 4001 steps 12.9 / 22.6 -> 7.0 / 10.9, 8192 steps 13 / 22 (with the
// cluster prefix) against 10.9 / 17.6; at 16,384 steps the three launches win, 14.4 / 24.9 against 18.6 / 35.8.
constexpr int64_t kScanShort = (int64_t)kClusterSteps * kClusterMax * kClusterThreads;

int launch_scan_short(const ScanArgs& a, int32_t dim, cudaStream_t s) {
    constexpr int64_t threads = (int64_t)kClusterMax * kClusterThreads;
    const int32_t per = (int32_t)((a.single_n_out + threads - 1) / threads);
    const int64_t ctas = (a.single_n_out + (int64_t)per * kClusterThreads - 1) / ((int64_t)per * kClusterThreads);
    unsigned c = 1;
    while (c < ctas) c *= 2;
    auto kernel = dim == 2 ? scan_short_kernel<2> : scan_short_kernel<3>;
    CUDA_TRY(launch_early_cluster(kernel, c, dim3(c), dim3(kClusterThreads), 0, s, a, per));
    return SPINSIM_OK;
}

// The tile prefixes: a warp per instance, or, where some instance has many tiles, a cluster per instance
// with about two tiles per thread of the longest (fewer CTAs where that would be many of them).  A warp
// takes 1.1 us for each 32 tiles of the longest instance from SU(2) partials, and 1.7 or 3 us from 2 x 2 or
// 3 x 3 products; a cluster kernel takes about 6 us and 0.5 us for each tile of its longest thread, in waves
// of three CTAs per SM (one of 6250 tiles 165 -> 10 us).  The shorter of the two is launched.
int launch_prefix(const ScanArgs& a, const ScanBuffers& b, const bool* has_dim, int sm, cudaStream_t s) {
    unsigned c = 1;
    while (c < (unsigned)kClusterMax && (int64_t)c * 2 * kClusterThreads < b.max_tiles &&
           (int64_t)2 * c * b.n_instances <= 16 * (int64_t)sm)
        c *= 2;
    const double per_chunk = a.partials ? 1.1 : has_dim[1] ? 3.0 : 1.7;
    const double by_warp = per_chunk * (double)((b.max_tiles + 31) / 32);
    const double per_thread = (double)((b.max_tiles + c * kClusterThreads - 1) / (c * kClusterThreads));
    const double waves = (double)(((int64_t)c * b.n_instances + 3 * sm - 1) / (3 * sm));
    const double by_cluster = (has_dim[0] + has_dim[1]) * waves * (6.0 + 0.5 * per_thread);
    if (by_warp <= by_cluster) {
        const unsigned warps_per_block = kScanBlock / 32;
        const unsigned grid = (unsigned)((b.n_instances + warps_per_block - 1) / warps_per_block);
        CUDA_TRY(launch_early(scan_prefix_kernel, dim3(grid), dim3(kScanBlock), 0, s, a));
        return SPINSIM_OK;
    }
    const dim3 grid(c * (unsigned)b.n_instances);
    if (has_dim[0]) CUDA_TRY(launch_early_cluster(scan_prefix_cluster_kernel<2>, c, grid, dim3(kClusterThreads), 0, s, a));
    if (has_dim[1]) CUDA_TRY(launch_early_cluster(scan_prefix_cluster_kernel<3>, c, grid, dim3(kClusterThreads), 0, s, a));
    return SPINSIM_OK;
}

// The state scan's launches (scan.cuh).  b.tiles == null: one instance (`single`, on the host) with
// implicit tiles.
// partials: the tensor-path time evolution has written each tile's warp partials into b.tile_product
// (the tile products kernels are then not launched).
// products: the time evolution has written the tile products themselves.
// rows (partials mode, may be null): each output step's operator as its SU(2) pair, which the apply
// reads in place of u.
int launch_scan(const Instance* inst_dev, const Instance* single, const ScanBuffers& b, const double* u, double* state,
                double* spin, cudaStream_t s, int stages = SCAN_ALL, double* total = nullptr, bool partials = false,
                const double* rows = nullptr, bool products = false) {
    if (b.n_tiles == 0) return SPINSIM_OK;
    ScanArgs a;
    memset(&a, 0, sizeof(a));
    a.instances = inst_dev;
    a.tiles = b.tiles;
    a.n_tiles = b.n_tiles;
    a.tile_begin = b.begin;
    a.tile_end = b.end;
    a.n_instances = b.n_instances;
    a.u = u;
    a.tile_product = b.tile_product;
    a.tile_prefix = b.tile_prefix;
    a.state = state;
    a.spin = spin;
    a.total = total;
    if (single) {
        a.single = *single;
        a.single_n_out = single->n_out;
        if (stages == SCAN_ALL && !total && single->n_out <= kScanShort) return launch_scan_short(a, single->dim, s);
    }
    a.partials = partials ? 1 : 0;
    a.rows = partials ? rows : nullptr;
    // tile kernels: one launch per spin dimension over its run of tiles
    const int64_t lo[2] = {0, b.tiles_half}, hi[2] = {b.tiles_half, b.n_tiles};
    const int warps[2] = {ScanShared<2>::kWarps, ScanShared<3>::kWarps};
    unsigned grid[2];
    for (int d = 0; d < 2; d++) {
        const int64_t w = (std::max<int64_t>(0, hi[d] - lo[d]) + kScanTilesPerWarp - 1) / kScanTilesPerWarp;
        grid[d] = (unsigned)((w + warps[d] - 1) / warps[d]);
    }
    constexpr int t2 = ScanShared<2>::kThreads, t3 = ScanShared<3>::kThreads;
    constexpr size_t m2 = ScanShared<2>::kBytes, m3 = ScanShared<3>::kBytes;
    int sm = 0;
    int rc = device_sm_count(&sm);
    if (rc) return rc;
    if (stages & SCAN_PREFIX) {
        if (grid[0] && !partials && !products)
            CUDA_TRY(launch_early(scan_products_kernel<2>, dim3(grid[0]), dim3(t2), m2, s, a, lo[0], hi[0]));
        if (grid[1] && !partials && !products)
            CUDA_TRY(launch_early(scan_products_kernel<3>, dim3(grid[1]), dim3(t3), m3, s, a, lo[1], hi[1]));
        const bool has_dim[2] = {grid[0] != 0, grid[1] != 0};
        rc = launch_prefix(a, b, has_dim, sm, s);
        if (rc) return rc;
    }
    if (stages & SCAN_APPLY) {  // persistent: at most the CTAs the device holds at once
        const int apply_warps[2] = {ApplyShared<2>::kWarps, ApplyShared<3>::kWarps};  // the same in both modes
        static_assert(ApplyShared<2, true>::kWarps == ApplyShared<2>::kWarps &&
                          ApplyShared<3, true>::kWarps == ApplyShared<3>::kWarps, "apply CTA sizes");
        unsigned agrid[2];
        for (int d = 0; d < 2; d++) {
            const int64_t groups = (std::max<int64_t>(0, hi[d] - lo[d]) + kScanTilesPerWarp - 1) / kScanTilesPerWarp;
            // resident CTAs per SM: shared memory allows 6 (d x d operators) or 10 and 7 (SU(2) pairs)
            const int64_t per_sm = a.rows == nullptr ? 6 : (d == 0 ? 10 : 7);
            agrid[d] = (unsigned)std::min<int64_t>((groups + apply_warps[d] - 1) / apply_warps[d], per_sm * sm);
        }
        // the first apply kernel waits for the prefixes; the second starts as the first's CTAs pass that
        // wait (launched early only when this call launched the prefix kernel just before)
        const bool early = (stages & SCAN_PREFIX) != 0;
        auto apply = [&](auto kernel, unsigned grid, int threads, size_t smem, int64_t tlo, int64_t thi,
                         int32_t after_prefix) -> cudaError_t {
            if (early) return launch_early(kernel, dim3(grid), dim3(threads), smem, s, a, tlo, thi, after_prefix);
            kernel<<<grid, threads, smem, s>>>(a, tlo, thi, after_prefix);
            return cudaGetLastError();
        };
        const int32_t second_after_prefix = agrid[0] ? 0 : 1;
        if (a.rows != nullptr) {
            if (agrid[0])
                CUDA_TRY(apply(scan_apply_kernel<2, true>, agrid[0], ApplyShared<2, true>::kThreads,
                               ApplyShared<2, true>::kBytes, lo[0], hi[0], 1));
            if (agrid[1])
                CUDA_TRY(apply(scan_apply_kernel<3, true>, agrid[1], ApplyShared<3, true>::kThreads,
                               ApplyShared<3, true>::kBytes, lo[1], hi[1], second_after_prefix));
        } else {
            if (agrid[0])
                CUDA_TRY(apply(scan_apply_kernel<2, false>, agrid[0], ApplyShared<2>::kThreads, ApplyShared<2>::kBytes,
                               lo[0], hi[0], 1));
            if (agrid[1])
                CUDA_TRY(apply(scan_apply_kernel<3, false>, agrid[1], ApplyShared<3>::kThreads, ApplyShared<3>::kBytes,
                               lo[1], hi[1], second_after_prefix));
        }
    }
    CUDA_TRY(cudaGetLastError());
    return SPINSIM_OK;
}

// early: the launch may start before the preceding kernel (the tensor path's constants) completes.
int launch_evolve(const spinsim_plan* p, EvolveArgs a, int64_t tiles, cudaStream_t s, bool early = false) {
    if (p->cta_tiles && !a.dmma_consts) return fail(SPINSIM_ERR_INVALID, "the tensor path's constants are missing");
    int64_t blocks = p->cta_tiles ? tiles : (tiles * 32 + p->block - 1) / p->block;
    if (a.tile_counter) {  // persistent: fill the device once, warps pull tiles from the queue
        const int64_t resident = (int64_t)p->sm_count * p->blocks_per_sm;
        blocks = std::min<int64_t>(blocks, resident);
    }
    if (blocks < 1) blocks = 1;
    if (blocks > 0x7fffffff) return fail(SPINSIM_ERR_INVALID, "launch too large");
    void* args[] = {&a};
    const size_t smem = (size_t)(p->block / 32) * p->smem_per_warp;
    if (early) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)blocks);
        cfg.blockDim = dim3(p->block);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = s;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        CUDA_TRY(cudaLaunchKernelExC(&cfg, p->func, args));
    } else {
        CUDA_TRY(cudaLaunchKernel(p->func, dim3((unsigned)blocks), dim3(p->block), args, smem, s));
    }
    return SPINSIM_OK;
}

// The tensor path's per-instance constants (evolve_dmma.cuh), which the time evolution then reads; for a
// single call also its descriptors (inst_out, field_out), from the arguments.
int launch_dmma_consts(EvolveArgs* a, DmmaConsts* out, int32_t n, Instance* inst_out, FieldDesc* field_out,
                       cudaStream_t s) {
    void* args[] = {a, &out, &n, &inst_out, &field_out};
    CUDA_TRY(cudaLaunchKernel(spinsim_kget_dmma_consts(), dim3((unsigned)n), dim3(kDmmaRecurrences), args, 0, s));
    a->dmma_consts = out;
    return SPINSIM_OK;
}

int check_field(const spinsim_plan* p, const spinsim_field* f) {
    if (!f) return fail(SPINSIM_ERR_INVALID, "field is null");
    if (p->desc.field_kind == SPINSIM_FIELD_TABLE && !f->tables)
        return fail(SPINSIM_ERR_INVALID, "a table field needs its device table array");
    if (p->desc.field_kind == SPINSIM_FIELD_TONES) {
        for (int c = 0; c < kMaxChannels; c++)
            if (f->tone_count[c] < 0 || f->tone_start[c] < 0) return fail(SPINSIM_ERR_INVALID, "negative tone count");
    }
    if (p->desc.field_kind == SPINSIM_FIELD_USER && f->n_params > 0 && !f->params)
        return fail(SPINSIM_ERR_INVALID, "sweep parameters missing");
    return SPINSIM_OK;
}
}  // namespace

// Whether an instance of an FP64 tone plan's launch (launch_steps output steps in all) runs on the tensor path.  Where
// the field lets it (tones_on_fp64_tensor_path), it does, but for launches of few output steps, of many fine steps with
// few tones each: the tensor path has four lanes for an output step, the per-sample kernel up to 32.  Whole calls, tensor
// path / per sample, spin one: 256 x 512 steps of 1 / 3 / 6 / 9 tones 85 / 49, 85 / 64, 86 / 83 and 85 / 98 us; of 3 tones
// 256 x 128 40 / 39, 1024 x 256 55 / 49, 2048 x 256 57 / 68, 256 x 8192 about 900 / 571.  A caller who fixed fewer lanes
// gets the tensor path's four (4 x 1000 steps of 3 tones: 129 us, per sample with 16 lanes 166).
static bool tensor_path_takes(const spinsim_plan* p, const FieldDesc& f, const Instance& inst, int64_t launch_steps) {
    if (!tones_on_fp64_tensor_path(f, inst)) return false;
    const int tones = f.tone_count[0] + f.tone_count[1] + f.tone_count[2];
    const bool all_lanes = p->m.lanes == 0 || p->m.lanes == 32;
    return !all_lanes || launch_steps > 1024 || inst.n_fine < 256 || tones > 4;
}

// ------------------------------------------------------------------ single instance
static int make_instance(const spinsim_plan* p, double t0, double dt_int, double dt_out, int64_t n_out,
                         const double* psi0, Instance* inst) {
    if (p->desc.spin_dim == 0) return fail(SPINSIM_ERR_INVALID, "a mixed plan evaluates batches only");
    if (n_out < 0) return fail(SPINSIM_ERR_INVALID, "negative number of output steps");
    if (!(dt_out > 0) || !(dt_int > 0)) return fail(SPINSIM_ERR_INVALID, "time steps must be positive");
    memset(inst, 0, sizeof(*inst));
    inst->t0 = t0;
    inst->dt_int = dt_int;
    inst->dt_out = dt_out;
    inst->n_out = n_out;
    const double k = floor(dt_out / dt_int + 0.5);
    if (!(k >= 0 && k < 2147483647.0)) return fail(SPINSIM_ERR_INVALID, "too many fine steps per output step");
    inst->n_fine = (int32_t)k;
    inst->dim = p->desc.spin_dim;
    if (psi0)
        for (int i = 0; i < 2 * inst->dim; i++) inst->psi0[i] = psi0[i];
    return SPINSIM_OK;
}

// Workspace of a single-instance call: the state scan's scratch (its descriptors are launch arguments, its
// tiles implicit) and, on the tensor path, its descriptors, constants and SU(2) rows.
static size_t single_workspace(int64_t n_out, bool with_scan, bool with_rows = false, bool tensor = false) {
    Carver c(nullptr);
    if (with_scan) {
        ScanBuffers b;
        carve_scan_single(c, n_out, 2, &b);
    }
    if (with_rows) c.take<double>(4 * (size_t)std::max<int64_t>(1, n_out));
    if (tensor) {
        c.take<Instance>(1);
        c.take<FieldDesc>(1);
        c.take<DmmaConsts>(1);
    }
    return c.used + 256;
}

extern "C" size_t spinsim_evaluate_workspace_size(const spinsim_plan* plan, int64_t n_out) {
    if (!plan || n_out < 0 || plan->desc.spin_dim == 0) return 0;
    // the tensor path's SU(2) rows for the scan (FP32-bulk), its descriptors and constants
    return single_workspace(n_out, true, plan->cta_tiles, plan->cta_tiles || plan->tensor);
}

static int evaluate_impl(const spinsim_plan* p, const spinsim_field* field, double t0, double dt_int, double dt_out,
                         int64_t n_out, const double* psi0, double* time, double* u, double* state, double* spin,
                         float* norms, void* ws, size_t ws_bytes, cudaStream_t s, bool with_scan,
                         const double* params = nullptr, int32_t n_params = 0) {
    if (!p) return fail(SPINSIM_ERR_INVALID, "plan is null");
    int rc = params ? (field ? SPINSIM_OK : fail(SPINSIM_ERR_INVALID, "field is null")) : check_field(p, field);
    if (rc) return rc;
    Instance inst;
    rc = make_instance(p, t0, dt_int, dt_out, n_out, psi0, &inst);
    if (rc) return rc;
    if (p->tensor && tensor_path_takes(p, *reinterpret_cast<const FieldDesc*>(field), inst, n_out)) p = p->tensor;
    if (n_out == 0) return SPINSIM_OK;
    if (!time || !u || (with_scan && !state)) return fail(SPINSIM_ERR_INVALID, "output pointer is null");
    if (with_scan && !psi0) return fail(SPINSIM_ERR_INVALID, "psi0 is null");
    if (!ws || ((uintptr_t)ws & 255)) return fail(SPINSIM_ERR_WORKSPACE, "workspace must be non-null and 256-byte aligned");
    const bool bulk = p->desc.precision == SPINSIM_PRECISION_FP32_BULK;
    const bool with_rows = with_scan && p->cta_tiles && bulk;
    const size_t need = single_workspace(n_out, with_scan, with_rows, p->cta_tiles);
    if (ws_bytes < need) return fail(SPINSIM_ERR_WORKSPACE, "workspace of %zu bytes is below the %zu needed", ws_bytes, need);

    Carver c(ws);
    ScanBuffers b;
    if (with_scan) carve_scan_single(c, n_out, inst.dim, &b);
    double* rows = with_rows ? c.take<double>(4 * (size_t)std::max<int64_t>(1, n_out)) : nullptr;

    EvolveArgs a;
    memset(&a, 0, sizeof(a));
    a.m = p->m;
    a.m.lanes = pick_lanes(p, n_out, inst.n_fine);
    a.single = inst;
    memcpy(&a.single_field, field, sizeof(FieldDesc));
    if (params) {
        a.n_single_params = n_params;
        memcpy(a.single_params, params, sizeof(double) * (size_t)n_params);
    }
    a.tiles = nullptr;
    const int per_tile = tile_intervals(p, a.m.lanes);
    a.n_tiles = (n_out + per_tile - 1) / per_tile;
    a.tile_counter = nullptr;
    a.time = time;
    a.u = u;
    a.step_norms = bulk ? norms : nullptr;
    // the tensor path writes the scan's tile partials as it goes (its CTA tiles are the scan tiles)
    const bool partials = with_scan && p->cta_tiles && bulk && n_out > kScanShort &&
                          tones_on_tensor_path(*reinterpret_cast<const FieldDesc*>(field), inst.dim);
    a.tile_partials = partials ? b.tile_product : nullptr;
    a.scan_begin = nullptr;
    a.rows = partials ? rows : nullptr;
    const bool products = with_scan && writes_products(p, a.m.lanes) && n_out > kScanShort;
    a.tile_products = products ? b.tile_product : nullptr;
    if (p->cta_tiles) {
        Instance* inst_dev = c.take<Instance>(1);
        FieldDesc* field_dev = c.take<FieldDesc>(1);
        rc = launch_dmma_consts(&a, c.take<DmmaConsts>(1), 1, inst_dev, field_dev, s);
        if (rc) return rc;
        a.instances = inst_dev;
        a.fields = field_dev;
    }
    rc = launch_evolve(p, a, a.n_tiles, s, p->cta_tiles);
    if (rc || !with_scan) return rc;
    return launch_scan(nullptr, &inst, b, u, state, spin, s, SCAN_ALL, nullptr, partials, a.rows, products);
}

extern "C" int spinsim_evaluate(const spinsim_plan* plan, const spinsim_field* field, double t0, double dt_int,
                                double dt_out, int64_t n_out, const double* psi0, double* time_dev, double* u_dev,
                                double* state_dev, double* spin_dev, void* workspace_dev, size_t workspace_bytes,
                                void* stream) {
    return evaluate_impl(plan, field, t0, dt_int, dt_out, n_out, psi0, time_dev, u_dev, state_dev, spin_dev, nullptr,
                         workspace_dev, workspace_bytes, (cudaStream_t)stream, true);
}

extern "C" int spinsim_evaluate_with_norms(const spinsim_plan* plan, const spinsim_field* field, double t0,
                                           double dt_int, double dt_out, int64_t n_out, const double* psi0,
                                           double* time_dev, double* u_dev, double* state_dev, double* spin_dev,
                                           float* step_norms_dev, void* workspace_dev, size_t workspace_bytes,
                                           void* stream) {
    return evaluate_impl(plan, field, t0, dt_int, dt_out, n_out, psi0, time_dev, u_dev, state_dev, spin_dev,
                         step_norms_dev, workspace_dev, workspace_bytes, (cudaStream_t)stream, true);
}

extern "C" int spinsim_evaluate_params(const spinsim_plan* plan, const double* params, int32_t n_params, double t0,
                                       double dt_int, double dt_out, int64_t n_out, const double* psi0,
                                       double* time_dev, double* u_dev, double* state_dev, double* spin_dev,
                                       float* step_norms_dev, void* workspace_dev, size_t workspace_bytes,
                                       void* stream) {
    if (!plan) return fail(SPINSIM_ERR_INVALID, "plan is null");
    if (plan->desc.field_kind != SPINSIM_FIELD_USER) return fail(SPINSIM_ERR_INVALID, "the plan has no user field");
    if (!params || n_params < 1 || n_params > kSingleParams)
        return fail(SPINSIM_ERR_INVALID, "between 1 and %d sweep parameters travel with the call", kSingleParams);
    spinsim_field field;
    memset(&field, 0, sizeof(field));
    return evaluate_impl(plan, &field, t0, dt_int, dt_out, n_out, psi0, time_dev, u_dev, state_dev, spin_dev,
                         step_norms_dev, workspace_dev, workspace_bytes, (cudaStream_t)stream, true, params, n_params);
}

extern "C" int spinsim_time_evolution(const spinsim_plan* plan, const spinsim_field* field, double t0, double dt_int,
                                      double dt_out, int64_t n_out, double* time_dev, double* u_dev,
                                      void* workspace_dev, size_t workspace_bytes, void* stream) {
    return evaluate_impl(plan, field, t0, dt_int, dt_out, n_out, nullptr, time_dev, u_dev, nullptr, nullptr, nullptr,
                         workspace_dev, workspace_bytes, (cudaStream_t)stream, false);
}

// ------------------------------------------------------------------ state / spin alone
static size_t state_ws(int64_t n_out) { return single_workspace(n_out, true); }

// The scan of one instance's operators in a workspace laid out as single_workspace's.
static int state_scan(int32_t dim, const double* u_dev, int64_t n_out, const double* psi0, double* state_dev,
                      double* spin_dev, double* total_dev, void* workspace, cudaStream_t s, int stages) {
    Instance inst;
    memset(&inst, 0, sizeof(inst));
    inst.dim = dim;
    inst.n_out = n_out;
    if (psi0)
        for (int i = 0; i < 2 * dim; i++) inst.psi0[i] = psi0[i];
    Carver c(workspace);
    ScanBuffers b;
    carve_scan_single(c, n_out, dim, &b);
    return launch_scan(nullptr, &inst, b, u_dev, state_dev, spin_dev, s, stages, total_dev);
}

extern "C" size_t spinsim_state_workspace_size(int32_t dim, int64_t n_out) {
    if ((dim != 2 && dim != 3) || n_out < 0) return 0;
    return state_ws(n_out);
}

extern "C" int spinsim_state(int32_t dim, const double* u_dev, int64_t n_out, const double* psi0, double* state_dev,
                             double* spin_dev, void* workspace_dev, size_t workspace_bytes, void* stream) {
    if (dim != 2 && dim != 3) return fail(SPINSIM_ERR_INVALID, "dim must be 2 or 3");
    if (n_out < 0) return fail(SPINSIM_ERR_INVALID, "negative length");
    if (n_out == 0) return SPINSIM_OK;
    if (!u_dev || !state_dev || !psi0) return fail(SPINSIM_ERR_INVALID, "null pointer");
    if (!workspace_dev || ((uintptr_t)workspace_dev & 255))
        return fail(SPINSIM_ERR_WORKSPACE, "workspace must be non-null and 256-byte aligned");
    if (workspace_bytes < state_ws(n_out)) return fail(SPINSIM_ERR_WORKSPACE, "workspace too small");
    return state_scan(dim, u_dev, n_out, psi0, state_dev, spin_dev, nullptr, workspace_dev, (cudaStream_t)stream,
                      SCAN_ALL);
}

// One evaluate() split into pieces (over launches or GPUs): each piece's product and, once the
// states entering the pieces are known, its states.  Both use the workspace layout of spinsim_state.
static int piece_scan(int32_t dim, const double* u_dev, int64_t n_out, const double* psi0, double* state_dev,
                      double* spin_dev, double* product_dev, void* workspace_dev, size_t workspace_bytes,
                      cudaStream_t s, int stages) {
    if (dim != 2 && dim != 3) return fail(SPINSIM_ERR_INVALID, "dim must be 2 or 3");
    if (n_out < 0) return fail(SPINSIM_ERR_INVALID, "negative length");
    if (n_out == 0) return SPINSIM_OK;
    if (!u_dev) return fail(SPINSIM_ERR_INVALID, "null pointer");
    if (!workspace_dev || ((uintptr_t)workspace_dev & 255))
        return fail(SPINSIM_ERR_WORKSPACE, "workspace must be non-null and 256-byte aligned");
    if (workspace_bytes < state_ws(n_out)) return fail(SPINSIM_ERR_WORKSPACE, "workspace too small");
    return state_scan(dim, u_dev, n_out, psi0, state_dev, spin_dev, product_dev, workspace_dev, s, stages);
}

extern "C" int spinsim_piece_product(int32_t dim, const double* u_dev, int64_t n_out, double* product_dev,
                                     void* workspace_dev, size_t workspace_bytes, void* stream) {
    if (!product_dev) return fail(SPINSIM_ERR_INVALID, "null pointer");
    return piece_scan(dim, u_dev, n_out, nullptr, nullptr, nullptr, product_dev, workspace_dev, workspace_bytes,
                      (cudaStream_t)stream, SCAN_PREFIX);
}

extern "C" int spinsim_piece_states(int32_t dim, const double* u_dev, int64_t n_out, const double* psi_in,
                                    double* state_dev, double* spin_dev, void* workspace_dev, size_t workspace_bytes,
                                    void* stream) {
    if (!psi_in || !state_dev) return fail(SPINSIM_ERR_INVALID, "null pointer");
    return piece_scan(dim, u_dev, n_out, psi_in, state_dev, spin_dev, nullptr, workspace_dev, workspace_bytes,
                      (cudaStream_t)stream, SCAN_APPLY);
}

static int spin_mean_chunks(int32_t members) { return std::min<int32_t>(members, 64); }

extern "C" size_t spinsim_spin_mean_workspace_size(int32_t members, int64_t n_out) {
    if (members <= 0 || n_out < 0) return 0;
    return (size_t)spin_mean_chunks(members) * (size_t)std::max<int64_t>(1, n_out) * 3 * sizeof(double) + 256;
}

extern "C" int spinsim_spin_mean(const double* spin_dev, int64_t first, int64_t stride, int32_t members, int64_t n_out,
                                 double* mean_dev, void* workspace_dev, size_t workspace_bytes, void* stream) {
    if (members <= 0 || n_out < 0 || first < 0 || stride < n_out)
        return fail(SPINSIM_ERR_INVALID, "members must be positive and stride at least n_out");
    if (n_out == 0) return SPINSIM_OK;
    if (!spin_dev || !mean_dev) return fail(SPINSIM_ERR_INVALID, "null pointer");
    if (!workspace_dev || ((uintptr_t)workspace_dev & 255))
        return fail(SPINSIM_ERR_WORKSPACE, "workspace must be non-null and 256-byte aligned");
    if (workspace_bytes < spinsim_spin_mean_workspace_size(members, n_out))
        return fail(SPINSIM_ERR_WORKSPACE, "workspace too small");
    cudaStream_t s = (cudaStream_t)stream;
    const int chunks = spin_mean_chunks(members);
    const int per_chunk = (members + chunks - 1) / chunks;
    double* partial = (double*)workspace_dev;
    dim3 grid((unsigned)((n_out + kMeanThreads - 1) / kMeanThreads), (unsigned)chunks);
    spin_mean_partial_kernel<<<grid, kMeanThreads, 0, s>>>(spin_dev, first, stride, members, per_chunk, n_out, partial);
    spin_mean_final_kernel<<<(unsigned)((3 * n_out + kMeanThreads - 1) / kMeanThreads), kMeanThreads, 0, s>>>(
        partial, chunks, members, n_out, mean_dev);
    CUDA_TRY(cudaGetLastError());
    return SPINSIM_OK;
}

extern "C" int spinsim_spin(int32_t dim, const double* state_dev, int64_t n_out, double* spin_dev, void* stream) {
    if (dim != 2 && dim != 3) return fail(SPINSIM_ERR_INVALID, "dim must be 2 or 3");
    if (n_out < 0) return fail(SPINSIM_ERR_INVALID, "negative length");
    if (n_out == 0) return SPINSIM_OK;
    if (!state_dev || !spin_dev) return fail(SPINSIM_ERR_INVALID, "null pointer");
    const unsigned grid = (unsigned)((n_out + 255) / 256);
    cudaStream_t s = (cudaStream_t)stream;
    if (dim == 2) spin_kernel<2><<<grid, 256, 0, s>>>(state_dev, n_out, spin_dev);
    else spin_kernel<3><<<grid, 256, 0, s>>>(state_dev, n_out, spin_dev);
    CUDA_TRY(cudaGetLastError());
    return SPINSIM_OK;
}

// ------------------------------------------------------------------ batches
struct spinsim_batch {
    const spinsim_plan* plan;
    Instance* inst_dev;
    FieldDesc* fields_dev;
    Tile* tiles_dev;
    int64_t n_tiles;
    Tile* tensor_tiles_dev = nullptr;  // FP64 tones: the tiles of the instances whose field the tensor path takes
    int64_t n_tensor_tiles = 0;        // (a launch of its own)
    int32_t* counter;                  // [2]: the two queues
    int lanes;
    float* step_norms = nullptr;  // FP32-bulk: per output step, the sum of |g|^2 over its fine steps
    ScanBuffers scan;  // every instance's scan tiles (both spins)
    bool partials = false;  // every instance takes the tensor path, which writes the scan's tile partials
    DmmaConsts* consts = nullptr;  // tensor path: per instance, written each launch by dmma_consts_kernel
    double* rows = nullptr;        // tensor path: each output step's operator as its SU(2) pair, for the scan
};

// The time evolution's tiles, ordered longest-first so that the long instances start early.  An
// instance's full tiles share one cost, so the (stable) order is found by sorting runs: each
// instance's full tiles as one run, its partial last tile as another.
// Only instances with tensor[i] == on (null: all).  Returns the number of tiles.
static int64_t fill_evolve_tiles(const spinsim_plan* p, const Instance* inst, int32_t n, int per_warp,
                                 const std::vector<char>* tensor, char on, Tile* out) {
    struct Run {
        double cost;
        int32_t instance;
        int32_t count;   // intervals per tile
        int64_t first;   // first interval of the run
        int64_t tiles;   // tiles in the run
    };
    std::vector<Run> runs;
    runs.reserve(2 * (size_t)n);
    for (int i = 0; i < n; i++) {
        if (tensor && (*tensor)[i] != on) continue;
        // a spin-one step costs about a spin-half one (SU(2) elements), more with a quadratic shift, and
        // its squarings with the eight-generator exponential
        const double step_cost =
            inst[i].dim == 2 ? 1.0 : p->m.expo_one == EXPO_LIE_TROTTER_8 ? 4.0 + 0.5 * p->m.hypercubes : 1.5;
        const int64_t full = inst[i].n_out / per_warp, rest = inst[i].n_out % per_warp;
        if (full) runs.push_back({step_cost * inst[i].n_fine * per_warp, i, per_warp, 0, full});
        if (rest) runs.push_back({step_cost * inst[i].n_fine * rest, i, (int32_t)rest, full * per_warp, 1});
    }
    std::stable_sort(runs.begin(), runs.end(), [](const Run& x, const Run& y) { return x.cost > y.cost; });
    int64_t at = 0;
    for (const Run& r : runs) {
        for (int64_t k = 0; k < r.tiles; k++) {
            Tile& t = out[at++];
            t.instance = r.instance;
            t.first = r.first + k * r.count;
            t.count = r.count;
        }
    }
    return at;
}

// Sizes and carves a batch's workspace (ws null: sizes only).  The tiles are written by
// batch_prepare, straight into the descriptors' staging image when there is one.
static int batch_layout(const spinsim_plan* p, const spinsim_instance* instances, int32_t n, int32_t n_fields,
                        void* ws, ScanPlan* sp, spinsim_batch* b, size_t* used, size_t* desc_bytes) {
    const Instance* inst = reinterpret_cast<const Instance*>(instances);
    int64_t total = 0;
    int max_fine = 1;
    for (int i = 0; i < n; i++) {
        if (inst[i].dim != 2 && inst[i].dim != 3) return fail(SPINSIM_ERR_INVALID, "instance %d: dim must be 2 or 3", i);
        if (p->desc.spin_dim && inst[i].dim != p->desc.spin_dim)
            return fail(SPINSIM_ERR_INVALID, "instance %d: dim %d does not match the plan", i, inst[i].dim);
        if (inst[i].n_out < 0 || inst[i].n_fine < 0) return fail(SPINSIM_ERR_INVALID, "instance %d: negative sizes", i);
        if (inst[i].field < 0 || inst[i].field >= n_fields) return fail(SPINSIM_ERR_INVALID, "instance %d: bad field index", i);
        total += inst[i].n_out;
        max_fine = std::max(max_fine, (int)inst[i].n_fine);
    }
    const int lanes = pick_lanes(p, total, max_fine);
    const int per_warp = tile_intervals(p, lanes);
    int64_t n_tiles = 0;
    int64_t n_tensor_tiles = 0;
    for (int i = 0; i < n; i++) {
        n_tiles += (inst[i].n_out + per_warp - 1) / per_warp;
        if (p->tensor) n_tensor_tiles += (inst[i].n_out + kDmmaTile - 1) / kDmmaTile;
    }
    count_scan_plan(inst, n, sp);

    // Workspace: every descriptor first (one block that a staged prepare uploads with one copy),
    // then the scratch.
    Carver c(ws);
    b->inst_dev = c.take<Instance>(std::max(1, n));
    b->fields_dev = c.take<FieldDesc>(std::max(1, n_fields));
    b->tiles_dev = c.take<Tile>(std::max<int64_t>(1, n_tiles));
    if (p->tensor) b->tensor_tiles_dev = c.take<Tile>(std::max<int64_t>(1, n_tensor_tiles));
    carve_scan_desc(c, *sp, &b->scan);
    if (desc_bytes) *desc_bytes = c.used;
    b->counter = c.take<int32_t>(2);
    carve_scan_scratch(c, b->scan.n_tiles, &b->scan);
    if (p->cta_tiles || p->tensor) b->consts = c.take<DmmaConsts>(std::max(1, n));
    if (p->cta_tiles) {
        b->rows = c.take<double>(4 * (size_t)std::max<int64_t>(1, total));
    }
    b->n_tiles = n_tiles;
    b->n_tensor_tiles = n_tensor_tiles;
    b->plan = p;
    b->lanes = lanes;
    *used = c.used + 256;
    return SPINSIM_OK;
}

extern "C" int spinsim_batch_describe(int32_t n, const double* t0, const double* t1, const double* dt_int,
                                      const double* dt_out, const int32_t* dim, const double* psi0,
                                      spinsim_instance* out, int64_t* totals) {
    if (n < 0 || (n && (!t0 || !t1 || !dt_int || !dt_out || !dim || !psi0 || !out)))
        return fail(SPINSIM_ERR_INVALID, "null argument");
    int64_t out_off = 0, u_off = 0, st_off = 0, steps = 0;
    for (int32_t i = 0; i < n; i++) {
        const int d = dim[i];
        if (d != 2 && d != 3) return fail(SPINSIM_ERR_INVALID, "instance %d: dim must be 2 or 3", i);
        double dti;
        int64_t n_out;
        int32_t k;
        int rc = spinsim_normalise_steps(t0[i], t1[i], dt_int[i], dt_out[i], &dti, &n_out, &k, nullptr);
        if (rc) return rc;
        spinsim_instance& s = out[i];
        memset(&s, 0, sizeof(s));
        s.t0 = t0[i];
        s.dt_int = dti;
        s.dt_out = dt_out[i];
        s.n_out = n_out;
        s.n_fine = k;
        s.dim = d;
        s.field = i;
        s.out_offset = out_off;
        s.u_offset = u_off;
        s.state_offset = st_off;
        for (int j = 0; j < 2 * d; j++) s.psi0[j] = psi0[6 * (int64_t)i + j];
        out_off += n_out;
        u_off += 2 * (int64_t)d * d * n_out;
        st_off += 2 * (int64_t)d * n_out;
        steps += n_out * k;
    }
    if (totals) {
        totals[0] = out_off;
        totals[1] = u_off;
        totals[2] = st_off;
        totals[3] = steps;
    }
    return SPINSIM_OK;
}

// ------------------------------------------------------------------ field packing (host only)
constexpr int64_t kTableDoubles = sizeof(spinsim_table) / sizeof(double);
static_assert(sizeof(spinsim_table) == 32, "table descriptor layout");
// Plan rows are 8 int64 each.  Per field a header row
//   {kind (1 table, 2 tones), n_rows, bias (double[8]*), gain (double[8]* or 0 = ones), data, n_data, counts, 0}
// where for tones data/n_data are the (w, A, phi) rows and counts points to int32 tone_start[8] then
// tone_count[8]; a table field's header is followed by n_rows channel rows
//   {channel, time (double*), amplitude (double*), size, order, zero_boundary, alias, 0}
// with alias = -1, or the index (within the field) of an earlier channel whose time array it shares.
extern "C" int64_t spinsim_pack_fields(int32_t n_fields, const int64_t* plan, int64_t n_plan_rows, double* host,
                                       int64_t host_doubles, uint64_t device_base, spinsim_field* fields_out) {
    if (n_fields < 0 || (n_fields && (!plan || !host || !fields_out)))
        return fail(SPINSIM_ERR_INVALID, "null argument");
    int64_t n_tables = 0;
    for (int64_t r = 0, f = 0; f < n_fields; f++) {
        if (r >= n_plan_rows) return fail(SPINSIM_ERR_INVALID, "field plan too short");
        const int64_t* h = plan + 8 * r;
        if (h[0] == 1) n_tables++;
        r += 1 + (h[0] == 1 ? h[1] : 0);
    }
    int64_t at = 8 * kTableDoubles * n_tables;  // table descriptors first
    if (at > host_doubles) return fail(SPINSIM_ERR_WORKSPACE, "staging too small for the field descriptors");
    memset(host, 0, (size_t)at * sizeof(double));
    int64_t row = 0, table_slot = 0;
    for (int32_t f = 0; f < n_fields; f++) {
        const int64_t* h = plan + 8 * row++;
        spinsim_field& out = fields_out[f];
        memset(&out, 0, sizeof(out));
        const double* bias = reinterpret_cast<const double*>(h[2]);
        const double* gain = reinterpret_cast<const double*>(h[3]);
        for (int c = 0; c < 8; c++) {
            out.bias[c] = bias ? bias[c] : 0.0;
            out.gain[c] = gain ? gain[c] : 1.0;
        }
        if (h[0] == 2) {  // tones
            const int64_t n = h[5];
            if (n < 0 || at + n > host_doubles) return fail(SPINSIM_ERR_WORKSPACE, "staging too small for field %d", f);
            const double* tones = reinterpret_cast<const double*>(h[4]);
            if (n) memcpy(host + at, tones, (size_t)n * sizeof(double));
            double rate = 1.0;
            for (int64_t k = 0; k + 2 < n; k += 3) rate = std::max(rate, fabs(tones[k]));
            out.n_params = rate < 1e18 ? (int64_t)ceil(rate) : (int64_t)1e18;
            const int32_t* counts = reinterpret_cast<const int32_t*>(h[6]);
            for (int c = 0; c < 8; c++) {
                out.tone_start[c] = counts[c];
                out.tone_count[c] = counts[8 + c];
            }
            out.tones = reinterpret_cast<const double*>(device_base + 8 * (uint64_t)at);
            at += n;
            continue;
        }
        if (h[0] != 1) return fail(SPINSIM_ERR_INVALID, "field %d: unknown kind %lld", f, (long long)h[0]);
        const int64_t n_rows = h[1];
        if (n_rows < 0 || n_rows > 8 || row + n_rows > n_plan_rows)
            return fail(SPINSIM_ERR_INVALID, "field %d: bad channel count", f);
        double* desc = host + 8 * kTableDoubles * table_slot;
        out.tables = reinterpret_cast<const spinsim_table*>(device_base + 8 * (uint64_t)(8 * kTableDoubles * table_slot));
        table_slot++;
        int64_t time_at[8];
        for (int64_t k = 0; k < n_rows; k++) {
            const int64_t* c = plan + 8 * (row + k);
            const int64_t ch = c[0], size = c[3], alias = c[6];
            if (ch < 0 || ch >= 8 || size < 0) return fail(SPINSIM_ERR_INVALID, "field %d: bad channel", f);
            if (alias >= 0 && (alias >= k || plan[8 * (row + alias) + 3] != size))
                return fail(SPINSIM_ERR_INVALID, "field %d: bad shared time array", f);
            if (at + (alias < 0 ? 2 : 1) * size > host_doubles)
                return fail(SPINSIM_ERR_WORKSPACE, "staging too small for field %d", f);
            if (alias < 0) {
                memcpy(host + at, reinterpret_cast<const double*>(c[1]), (size_t)size * sizeof(double));
                time_at[k] = at;
                at += size;
            } else {
                time_at[k] = time_at[alias];
            }
            memcpy(host + at, reinterpret_cast<const double*>(c[2]), (size_t)size * sizeof(double));
            spinsim_table t;
            t.time = reinterpret_cast<const double*>(device_base + 8 * (uint64_t)time_at[k]);
            t.amplitude = reinterpret_cast<const double*>(device_base + 8 * (uint64_t)at);
            t.size = size;
            t.order = (int32_t)c[4];
            t.zero_boundary = (int32_t)c[5];
            memcpy(desc + kTableDoubles * ch, &t, sizeof(t));
            at += size;
        }
        row += n_rows;
    }
    return at;
}

extern "C" size_t spinsim_batch_workspace_size(const spinsim_plan* plan, const spinsim_instance* instances,
                                               int32_t n_instances, int32_t n_fields) {
    if (!plan || (!instances && n_instances) || n_instances < 0 || n_fields < 0) return 0;
    ScanPlan sp;
    spinsim_batch b;
    size_t used = 0;
    if (batch_layout(plan, instances, n_instances, n_fields, nullptr, &sp, &b, &used, nullptr)) return 0;
    return used;
}

extern "C" size_t spinsim_batch_staging_size(const spinsim_plan* plan, const spinsim_instance* instances,
                                             int32_t n_instances, int32_t n_fields) {
    if (!plan || (!instances && n_instances) || n_instances < 0 || n_fields < 0) return 0;
    ScanPlan sp;
    spinsim_batch b;
    size_t used = 0, desc = 0;
    if (batch_layout(plan, instances, n_instances, n_fields, nullptr, &sp, &b, &used, &desc)) return 0;
    return desc;
}

// Copy `bytes` from host `src` to the descriptor at `dst`: into the staging image of the
// descriptor block (at the same offset from its start as dst from the workspace), or directly.
static int put_desc(void* dst, const void* src, size_t bytes, void* ws, char* staging, cudaStream_t s) {
    if (!bytes) return SPINSIM_OK;
    if (staging) {
        memcpy(staging + ((char*)dst - (char*)ws), src, bytes);
        return SPINSIM_OK;
    }
    return upload(dst, src, bytes, s);
}

static int batch_prepare(const spinsim_plan* plan, const spinsim_instance* instances, int32_t n_instances,
                         const spinsim_field* fields, int32_t n_fields, void* workspace_dev, size_t workspace_bytes,
                         void* host_staging, size_t staging_bytes, cudaStream_t s, spinsim_batch** out) {
    if (!plan || !out || (n_instances && (!instances || !fields))) return fail(SPINSIM_ERR_INVALID, "null argument");
    *out = nullptr;
    if (!workspace_dev || ((uintptr_t)workspace_dev & 255))
        return fail(SPINSIM_ERR_WORKSPACE, "workspace must be non-null and 256-byte aligned");
    for (int i = 0; i < n_fields; i++) {
        int rc = check_field(plan, fields + i);
        if (rc) return rc;
    }
    ScanPlan sp;
    spinsim_batch* b = new spinsim_batch();
    size_t used = 0, desc = 0;
    int rc = batch_layout(plan, instances, n_instances, n_fields, workspace_dev, &sp, b, &used, &desc);
    if (!rc && workspace_bytes < used) rc = fail(SPINSIM_ERR_WORKSPACE, "workspace of %zu bytes is below the %zu needed", workspace_bytes, used);
    if (!rc && host_staging && staging_bytes < desc)
        rc = fail(SPINSIM_ERR_WORKSPACE, "staging of %zu bytes is below the %zu needed", staging_bytes, desc);
    char* st = (char*)host_staging;
    void* ws = workspace_dev;
    if (!rc) rc = put_desc(b->inst_dev, instances, sizeof(Instance) * n_instances, ws, st, s);
    if (!rc) rc = put_desc(b->fields_dev, fields, sizeof(FieldDesc) * n_fields, ws, st, s);
    if (!rc) {
        // The tile lists: written in place in the staging image, else built here and uploaded.
        const Instance* inst = reinterpret_cast<const Instance*>(instances);
        const int per_warp = tile_intervals(plan, b->lanes);
        std::vector<char> on_path;  // FP64 tones: which instances the tensor path takes
        int64_t total = 0;
        for (int i = 0; i < n_instances; i++) total += inst[i].n_out;
        if (plan->tensor)
            for (int i = 0; i < n_instances; i++)
                on_path.push_back(tensor_path_takes(plan, reinterpret_cast<const FieldDesc*>(fields)[inst[i].field], inst[i], total));
        std::vector<Tile> evolve_tiles, tensor_tiles, scan_tiles;
        std::vector<int32_t> begin, end;
        Tile *et, *tt, *stl;
        int32_t *bg, *en;
        if (st) {
            et = reinterpret_cast<Tile*>(st + ((char*)b->tiles_dev - (char*)ws));
            tt = plan->tensor ? reinterpret_cast<Tile*>(st + ((char*)b->tensor_tiles_dev - (char*)ws)) : nullptr;
            stl = reinterpret_cast<Tile*>(st + ((char*)b->scan.tiles - (char*)ws));
            bg = reinterpret_cast<int32_t*>(st + ((char*)b->scan.begin - (char*)ws));
            en = reinterpret_cast<int32_t*>(st + ((char*)b->scan.end - (char*)ws));
        } else {
            evolve_tiles.resize((size_t)b->n_tiles);
            tensor_tiles.resize((size_t)b->n_tensor_tiles);
            scan_tiles.resize((size_t)sp.n_tiles);
            begin.resize((size_t)n_instances);
            end.resize((size_t)n_instances);
            et = evolve_tiles.data();
            tt = tensor_tiles.data();
            stl = scan_tiles.data();
            bg = begin.data();
            en = end.data();
        }
        if (plan->tensor) {
            b->n_tensor_tiles = fill_evolve_tiles(plan->tensor, inst, n_instances, kDmmaTile, &on_path, 1, tt);
            b->n_tiles = fill_evolve_tiles(plan, inst, n_instances, per_warp, &on_path, 0, et);
        } else {
            fill_evolve_tiles(plan, inst, n_instances, per_warp, nullptr, 0, et);
        }
        fill_scan_plan(inst, n_instances, stl, bg, en);
        if (st) {
            rc = upload(ws, st, desc, s);
        } else {
            rc = upload(b->tiles_dev, et, sizeof(Tile) * (size_t)b->n_tiles, s);
            if (!rc) rc = upload(b->tensor_tiles_dev, tt, sizeof(Tile) * (size_t)b->n_tensor_tiles, s);
            if (!rc) rc = upload(b->scan.tiles, stl, sizeof(Tile) * (size_t)sp.n_tiles, s);
            if (!rc) rc = upload(b->scan.begin, bg, sizeof(int32_t) * (size_t)n_instances, s);
            if (!rc) rc = upload(b->scan.end, en, sizeof(int32_t) * (size_t)n_instances, s);
            // pageable sources: the copies have read them when cudaMemcpyAsync returns
        }
    }
    if (rc) {
        delete b;
        return rc;
    }
    if (plan->cta_tiles) {
        const Instance* inst = reinterpret_cast<const Instance*>(instances);
        const FieldDesc* fd = reinterpret_cast<const FieldDesc*>(fields);
        b->partials = true;
        for (int i = 0; i < n_instances && b->partials; i++)
            b->partials = tones_on_tensor_path(fd[inst[i].field], inst[i].dim);
    }
    *out = b;
    return SPINSIM_OK;
}

extern "C" int spinsim_batch_prepare(const spinsim_plan* plan, const spinsim_instance* instances, int32_t n_instances,
                                     const spinsim_field* fields, int32_t n_fields, void* workspace_dev,
                                     size_t workspace_bytes, void* stream, spinsim_batch** out) {
    return batch_prepare(plan, instances, n_instances, fields, n_fields, workspace_dev, workspace_bytes, nullptr, 0,
                         (cudaStream_t)stream, out);
}

extern "C" int spinsim_batch_prepare_staged(const spinsim_plan* plan, const spinsim_instance* instances,
                                            int32_t n_instances, const spinsim_field* fields, int32_t n_fields,
                                            void* workspace_dev, size_t workspace_bytes, void* host_staging,
                                            size_t staging_bytes, void* stream, spinsim_batch** out) {
    if (!host_staging) return fail(SPINSIM_ERR_INVALID, "staging buffer is null");
    return batch_prepare(plan, instances, n_instances, fields, n_fields, workspace_dev, workspace_bytes, host_staging,
                         staging_bytes, (cudaStream_t)stream, out);
}

extern "C" int spinsim_batch_launch(const spinsim_batch* b, double* time_dev, double* u_dev, double* state_dev,
                                    double* spin_dev, void* stream) {
    if (!b) return fail(SPINSIM_ERR_INVALID, "batch is null");
    if (b->n_tiles + b->n_tensor_tiles == 0) return SPINSIM_OK;
    if (!time_dev || !u_dev) return fail(SPINSIM_ERR_INVALID, "output pointer is null");
    cudaStream_t s = (cudaStream_t)stream;
    const spinsim_plan* p = b->plan;
    CUDA_TRY(cudaMemsetAsync(b->counter, 0, 2 * sizeof(int32_t), s));
    EvolveArgs a;
    memset(&a, 0, sizeof(a));
    a.instances = b->inst_dev;
    a.fields = b->fields_dev;
    a.time = time_dev;
    a.u = u_dev;
    a.step_norms = p->desc.precision == SPINSIM_PRECISION_FP32_BULK ? b->step_norms : nullptr;
    a.tile_partials = b->partials ? b->scan.tile_product : nullptr;  // the same kernel work with or without the scan
    a.rows = b->partials ? b->rows : nullptr;
    // the scan's tile products, when every launch of the time evolution writes its own
    const bool products = (b->n_tensor_tiles == 0 || writes_products(p->tensor, 1)) &&
                          (b->n_tiles == 0 || writes_products(p, b->lanes));
    a.tile_products = products ? b->scan.tile_product : nullptr;
    a.scan_begin = b->scan.begin;
    if (b->consts != nullptr && b->scan.n_instances > 0 && (p->cta_tiles || b->n_tensor_tiles > 0)) {
        int rc = launch_dmma_consts(&a, b->consts, b->scan.n_instances, nullptr, nullptr, s);
        if (rc) return rc;
    }
    auto evolve = [&](const spinsim_plan* q, int lanes, const Tile* tiles, int64_t n_tiles, int32_t* counter) {
        if (n_tiles == 0) return (int)SPINSIM_OK;
        a.m = q->m;
        a.m.lanes = lanes;
        a.tiles = tiles;
        a.n_tiles = n_tiles;
        a.tile_counter = counter;
        return launch_evolve(q, a, n_tiles, s, q->cta_tiles);  // early behind the tensor path's constants
    };
    int rc = evolve(p->tensor, 1, b->tensor_tiles_dev, b->n_tensor_tiles, b->counter + 1);
    if (!rc) rc = evolve(p, b->lanes, b->tiles_dev, b->n_tiles, b->counter);
    if (rc || !state_dev) return rc;
    rc = launch_scan(b->inst_dev, nullptr, b->scan, u_dev, state_dev, spin_dev, s, SCAN_ALL, nullptr, b->partials, a.rows,
                     products);
    return rc;
}

extern "C" int spinsim_batch_set_step_norms(spinsim_batch* b, float* step_norms_dev) {
    if (!b) return fail(SPINSIM_ERR_INVALID, "batch is null");
    b->step_norms = step_norms_dev;
    return SPINSIM_OK;
}

extern "C" int spinsim_batch_get_info(const spinsim_batch* b, spinsim_batch_info* info) {
    if (!b || !info) return fail(SPINSIM_ERR_INVALID, "null argument");
    info->tiles = b->n_tiles + b->n_tensor_tiles;
    info->scan_tiles = b->scan.n_tiles;
    const bool tensor_only = b->n_tiles == 0 && b->n_tensor_tiles > 0;
    info->lanes = tensor_only ? 1 : b->lanes;
    info->tile_intervals = tensor_only ? kDmmaTile : tile_intervals(b->plan, b->lanes);
    info->scan_partials = b->partials ? 1 : 0;
    info->reserved = 0;
    return SPINSIM_OK;
}

extern "C" int spinsim_batch_destroy(spinsim_batch* b) {
    delete b;
    return SPINSIM_OK;
}

// ------------------------------------------------------------------ diagnostics
namespace {
__device__ double g_fma_sink;

// Eight independent FMA chains per thread: the issue-rate ceiling of the FP64 or FP32 pipe.
template <typename T>
__global__ void __launch_bounds__(256) fma_peak_kernel(int iters, T seed) {
    T a0 = seed + (T)threadIdx.x, a1 = a0 + (T)1, a2 = a0 + (T)2, a3 = a0 + (T)3;
    T a4 = a0 + (T)4, a5 = a0 + (T)5, a6 = a0 + (T)6, a7 = a0 + (T)7;
    const T b = (T)0.999999, c = (T)1e-3;
    for (int i = 0; i < iters; i++) {
#pragma unroll
        for (int u = 0; u < 4; u++) {
            a0 = fma(a0, b, c); a1 = fma(a1, b, c); a2 = fma(a2, b, c); a3 = fma(a3, b, c);
            a4 = fma(a4, b, c); a5 = fma(a5, b, c); a6 = fma(a6, b, c); a7 = fma(a7, b, c);
        }
    }
    const T s = ((a0 + a1) + (a2 + a3)) + ((a4 + a5) + (a6 + a7));
    if (s == (T)-12345.0) g_fma_sink = (double)s;
}
}  // namespace

extern "C" int spinsim_fma_peak(int32_t precision, double* flops, void* stream) {
    if (precision != 0 && precision != 1) return fail(SPINSIM_ERR_INVALID, "precision must be 0 (FP64) or 1 (FP32)");
    int dev = 0, sms = 0;
    CUDA_TRY(cudaGetDevice(&dev));
    CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int iters = precision == 0 ? 2048 : 4096;
    const unsigned blocks = (unsigned)sms * 8, threads = 256;
    cudaStream_t s = (cudaStream_t)stream;
    if (precision == 0) fma_peak_kernel<double><<<blocks, threads, 0, s>>>(iters, 1.0);
    else fma_peak_kernel<float><<<blocks, threads, 0, s>>>(iters, 1.0f);
    CUDA_TRY(cudaGetLastError());
    if (flops) *flops = (double)blocks * threads * iters * 4 * 8 * 2;
    return SPINSIM_OK;
}

// ------------------------------------------------------------------ state propagation without allocation
// spinsim_state_static: spinsim_state with its scratch in a fixed device array owned by this
// library, for callers that may not allocate device memory themselves.  Such callers exist: a plugin
// that only ever receives device buffers from a host application which owns every allocation (its
// own allocator or a fixed memory pool), or a loop that must not pay the device-wide
// synchronisation a cudaMalloc/cudaFree implies.  They still pass the inputs (operators, initial
// state) and the outputs (state, spin); only the scan's scratch comes from here.
//
// The array below is a file-scope __device__ variable: every GPU that loads this library holds
// kStaticStateBytes of it until the process exits.  Host code must not hand the symbol itself to a
// kernel (on the host it names a host-side stand-in, not device memory), so the first call on each
// device, with that device current, asks the runtime for its device address (cudaGetSymbolAddress)
// and keeps it.  That first call may load the module; make it before any stream capture.  All calls
// on a device share the one array, so calls whose work overlaps on the GPU (other streams, other host
// threads) race and must be serialised by the caller.  Everything the scan reads from the array is
// written earlier in the same call (the instance descriptor, tile products, then tile prefixes), so no
// clearing between calls is needed.
namespace {
constexpr int64_t kStaticStateMaxSteps = 262144;  // 2^18 output steps, either spin
constexpr size_t kStaticStateBytes = (size_t)5 << 20;
constexpr int kStaticMaxDevices = 64;
__device__ __align__(256) unsigned char g_state_scratch[kStaticStateBytes];
std::mutex g_state_scratch_mutex;
void* g_state_scratch_ptr[kStaticMaxDevices] = {};

int state_scratch_address(void** out) {
    int dev = 0;
    CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kStaticMaxDevices) return fail(SPINSIM_ERR_INVALID, "device %d out of range", dev);
    std::lock_guard<std::mutex> lock(g_state_scratch_mutex);
    if (!g_state_scratch_ptr[dev]) {
        void* p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_state_scratch);
        if (e != cudaSuccess || !p)
            return fail(SPINSIM_ERR_CUDA, "cudaGetSymbolAddress of the state scratch failed: %s", cudaGetErrorString(e));
        g_state_scratch_ptr[dev] = p;
    }
    *out = g_state_scratch_ptr[dev];
    return SPINSIM_OK;
}
}  // namespace

extern "C" int64_t spinsim_state_static_max_steps(void) { return kStaticStateMaxSteps; }

extern "C" int spinsim_state_static(int32_t dim, const double* u_dev, int64_t n_out, const double* psi0,
                                    double* state_dev, double* spin_dev, void* stream) {
    if (dim != 2 && dim != 3) return fail(SPINSIM_ERR_INVALID, "dim must be 2 or 3");
    if (n_out < 0) return fail(SPINSIM_ERR_INVALID, "negative length");
    if (n_out > kStaticStateMaxSteps)
        return fail(SPINSIM_ERR_INVALID,
                    "spinsim_state_static handles at most %lld output steps (got %lld); use spinsim_state "
                    "with a caller-allocated workspace",
                    (long long)kStaticStateMaxSteps, (long long)n_out);
    if (n_out == 0) return SPINSIM_OK;
    if (!u_dev || !state_dev || !psi0) return fail(SPINSIM_ERR_INVALID, "null pointer");
    if (state_ws(n_out) > kStaticStateBytes)
        return fail(SPINSIM_ERR_INVALID, "state scratch of %zu bytes exceeds the static %zu", state_ws(n_out),
                    kStaticStateBytes);
    void* scratch = nullptr;
    int rc = state_scratch_address(&scratch);
    if (rc) return rc;
    return state_scan(dim, u_dev, n_out, psi0, state_dev, spin_dev, nullptr, scratch, (cudaStream_t)stream, SCAN_ALL);
}
