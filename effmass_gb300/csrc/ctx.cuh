// ctx.cuh — internal state of a context (hpsi_ctx) and of its bound
// k-points, shared by the C-ABI translation units (hpsi_api.cu, batch.cu).
#pragma once

#include <cstdarg>
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <map>
#include <string>
#include <vector>

#include "../../include/hpsi_gb300.h"
#include "d64_gemm.cuh"
#include "kernels.cuh"
#include "tc_gemm.cuh"

// A device buffer kept when a slot is rebound, for the next binding
struct Spare {
    void* p = nullptr;
    size_t bytes = 0;
};
// What a context keeps at most, all spares together.  Larger buffers go back to the
// device at once (their builds take longer than cudaMalloc and cudaFree), and so
// does a spare that no call took between two rebindings.
constexpr size_t kSpareMax = 64ull << 20;

struct KSlot {
    bool valid = false;
    int npw = 0;
    double kf[3] = {0, 0, 0};
    // the binding's tables, d_kin to d_lam, in one allocation
    unsigned char* mem = nullptr;
    size_t mem_cap = 0;
    double* d_kin = nullptr;
    double* d_kvec = nullptr;
    int* d_g = nullptr;
    double* d_q = nullptr;
    double* d_trig = nullptr;
    double* d_ylm = nullptr;   // ylm, yth, yph consecutive
    double* d_beta = nullptr;  // beta, dbeta consecutive
    double* d_dbeta0 = nullptr;
    double2* d_sf = nullptr;
    int nxs = 0;
    bool aliased = false;          // two G-vectors map to one grid point (the scatter keeps the last)
    int* d_plane = nullptr;    // plane_x[nxs], plane_off[nxs+1], ent_ig[npw], ent_jk[npw]
    int P = 0;
    std::vector<ProjRow> rows;     // host copy of d_rows
    ProjRow* d_rows = nullptr;
    double* d_lam = nullptr;
    // projector matrices: rows [0, P), and with dbeta tables room for the 3 P
    // derivative rows behind them (filled on first use: pr*_grad)
    double2* pr64 = nullptr;
    bool pr64_built = false, pr64_grad = false;  // rows [0, P) and the derivative rows hold their values
    // exponents of pr64 for the digit split (d64_scale_at), of the first P rows (H) and
    // of all 4 P (gradient), in pr64's allocation
    int* d64_exp[2] = {nullptr, nullptr};
    bool d64_exp_set[2] = {false, false};
    float2* pr32 = nullptr;
    bool pr32_built = false, pr32_grad = false;
    size_t pr_bytes[2] = {0, 0};   // allocation sizes of pr64, pr32
    size_t tc_bytes[2] = {0, 0};   // and of tc_mem
    // tensor-core H|psi>: generator tables of the projector operands, one set
    // per split format (0 FP16, 1 BF16), built from the FP64 tables on first
    // use and kept until the slot is rebound (batch plans hold pointers into
    // them); tc_proj and tc_expand carry only their K depth and row factors.
    // tc_fmt: the format of the last preparation, which the call that follows
    // it uses.
    int tc_fmt = -1;
    unsigned char* tc_mem[2] = {nullptr, nullptr};
    TcGen tcgen[2];
    TcOperand tc_proj[2], tc_expand[2];
    int tcg_fmt = -1;              // gradient operands (4P-row projection, per-direction expansion)
    bool tcg_built = false;
    unsigned char* tcg_mem = nullptr;
    TcOperand tcg_proj, tcg_exp[3];
    long gen = 0;                  // binding generation: changes when the slot is rebound
    double2* hess64 = nullptr;     // projector second derivatives [6][P][npw] (Hessian), per precision
    float2* hess32 = nullptr;
    bool hess64_built = false, hess32_built = false;
};

// Whether work queued on st is recorded into a graph instead of run.  A first-use
// build that is recorded is not marked as built: the next eager call cannot know
// whether the graph has been launched, and builds again.
inline bool capturing(cudaStream_t st)
{
    cudaStreamCaptureStatus s = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &s) != cudaSuccess) {
        cudaGetLastError();  // the legacy stream while another one captures
        return false;
    }
    return s != cudaStreamCaptureStatusNone;
}

template <typename T>
inline cudaError_t dalloc(T** p, size_t count)
{
    *p = nullptr;
    if (count == 0) return cudaSuccess;
    return cudaMalloc((void**)p, count * sizeof(T));
}

template <typename T>
inline void dfree(T*& p)
{
    if (p) cudaFree(p);
    p = nullptr;
}

inline void slot_free(KSlot& s)
{
    dfree(s.mem);
    dfree(s.pr64); dfree(s.pr32); dfree(s.tc_mem[0]); dfree(s.tc_mem[1]); dfree(s.tcg_mem); dfree(s.hess64);
    dfree(s.hess32);
    s = KSlot();
}

struct hpsi_ctx {
    int dev = 0;
    int n1 = 0, n2 = 0, n3 = 0;
    double omega = 0;
    int natom = 0, nrad = 0, nq_max = 0, lmax = 0;
    bool have_dbeta = true;
    std::vector<int> atom_species, rad_off, rad_l, rad_nq;
    std::vector<double> tau, rad_lam, rad_dq, rad_qmax;
    double* d_tables = nullptr;   // beta then dbeta, [2][nrad][nq_max]
    int* d_rad_nq = nullptr;
    double* d_rad_dq = nullptr;
    double* d_tau = nullptr;
    double* d_v64 = nullptr;
    float* d_v32 = nullptr;
    float* d_dv32 = nullptr;      // V64 - V32 per grid point (the energy sums' FP64 correction)
    int4* d_tw64 = nullptr;       // twiddles x, y, z consecutive (Q62 words)
    float2* d_tw32 = nullptr;
    FftLen L[3];
    std::map<int, KSlot> slots;
    // projector buffers of the last binding that was replaced: pr64, pr32, tc_mem[0], [1]
    Spare spare[4];
    // projector rows and strengths (the same for every k-point), and the largest q
    // that every radial table covers
    std::vector<ProjRow> proj_rows;
    std::vector<double> proj_lam;
    D64Rows proj_groups;          // their groups by radial function (arrays in d_groups)
    int* d_groups = nullptr;
    double q_safe = 0;
    unsigned char* stage = nullptr;  // pinned staging of hpsi_set_kpoint
    size_t stage_size = 0;
    unsigned char* ws = nullptr;
    size_t ws_size = 0;
    // the first workspace stays with the context: freeing it when a call needs more
    // would cost that call the time of a cudaFree (50-80 us)
    unsigned char* ws_first = nullptr;
    size_t ws_first_size = 0;
    // workspace of the FP64 GEMMs on the tensor cores (set per call): behind the call's
    // own in ws where that has room, else d64_mem.  A call that cannot have it runs the
    // SIMT GEMMs, and d64_mem goes back to the device when anything else finds no room.
    unsigned char* d64_ws = nullptr;
    size_t d64_size = 0;
    unsigned char* d64_mem = nullptr;
    size_t d64_cap = 0;
    // the smallest workspace that the device had no room for, and its free bytes then:
    // not asked for again before more is free
    size_t d64_refused = SIZE_MAX, d64_refused_free = 0;
    // test hooks (hpsi_selftest_memory): largest d64_mem granted, allocations that are
    // to find no room, and allocations of d64_mem tried
    size_t test_d64_room = SIZE_MAX;
    int test_oom = 0;
    long d64_tries = 0;
    // tensor-core work of an FP64 call whose outcome (d_err) no call has read yet, and
    // its stream: every call that synchronises that stream reads it (finish)
    bool d64_ran = false;
    cudaStream_t d64_stream = nullptr;
    Prof prof;
    int* d_err = nullptr;         // device-side error flag of the bounded waits (tcgen05 GEMMs)
    // side stream of the FP64 and tensor-core H|psi>: the projection chain runs there
    // beside the FFT passes (fork/join by events on the caller's stream)
    cudaStream_t side = nullptr;
    cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
    // copy stream of hpsi_apply with host buffers: the H2D copy of hpsi, which
    // only the tensor-core expansion reads, runs beside the FFT passes
    cudaStream_t copy = nullptr;
    cudaEvent_t ev_copy_after = nullptr, ev_copy_done = nullptr;
    // hpsi_apply with host buffers on the tensor-core path: hpsi moves in and
    // out in two G halves (uploads on the copy stream, the first half's
    // download on the side stream beside the second half's expansion)
    cudaEvent_t ev_half_in[2] = {nullptr, nullptr}, ev_half_exp = nullptr, ev_half_out = nullptr;
    cudaEvent_t ev_psi_in[2] = {nullptr, nullptr};  // psi's two band halves on the copy stream
    long gen_counter = 0;         // source of KSlot::gen
    double* d_hess = nullptr;     // Hessian radial tables [nrad][3][hess_nq] (F0, F1, F3), raw
    int hess_nq = 0;
    double hess_dq = 0.0;
    std::vector<char> hess_set;   // per radial function: tables given
    std::string err;
};

// Message of the last failure that had no context to hold it (hpsi_ctx_create,
// batch plans).
extern thread_local std::string g_last_error;

inline int fail(hpsi_ctx* c, int code, const char* fmt, ...)
{
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    if (c) c->err = buf;
    else g_last_error = buf;
    return code;
}

#define CUDA_TRY(ctx, expr)                                                                             \
    do {                                                                                                \
        cudaError_t e_ = (expr);                                                                        \
        if (e_ != cudaSuccess)                                                                          \
            return fail(ctx, e_ == cudaErrorMemoryAllocation ? HPSI_ERR_OOM : HPSI_ERR_CUDA, "%s: %s (%s:%d)", \
                        #expr, cudaGetErrorString(e_), __FILE__, __LINE__);                             \
    } while (0)

// Workspace carving: each piece 256-byte aligned.
struct Carver {
    size_t off = 0;
    template <typename T>
    size_t take(size_t count)
    {
        size_t o = off;
        off += ((count * sizeof(T)) + 255) / 256 * 256;
        return o;
    }
};

// Give memory that only makes calls faster back to the device; false if there is none.
inline bool release_optional(hpsi_ctx* c)
{
    bool any = c->d64_mem != nullptr;
    if (c->d64_ws == c->d64_mem) c->d64_ws = nullptr;
    dfree(c->d64_mem);
    c->d64_cap = 0;
    for (Spare& p : c->spare) {
        any = any || p.p;
        dfree(p.p);
        p.bytes = 0;
    }
    return any;
}

// cudaMalloc that asks for optional memory back before it reports that there is no room
template <typename T>
inline cudaError_t dev_malloc(hpsi_ctx* c, T** p, size_t bytes)
{
    *p = nullptr;
    cudaError_t e = c->test_oom > 0 ? cudaErrorMemoryAllocation : cudaMalloc((void**)p, bytes);
    if (c->test_oom > 0) --c->test_oom;
    if (e != cudaErrorMemoryAllocation || !release_optional(c)) return e;
    cudaGetLastError();
    return cudaMalloc((void**)p, bytes);
}

// Empty slot s for a new binding.  The tables' allocation stays with it, its projector
// buffers stay with the context as spares.  The caller has synchronised the device.
inline void slot_reset(hpsi_ctx* c, KSlot& s)
{
    size_t kept = 0;
    auto keep = [&](Spare& to, auto*& p, size_t bytes) {
        dfree(to.p);
        to.bytes = 0;
        if (!p || kept + bytes > kSpareMax) return;
        to = Spare{p, bytes};
        kept += bytes;
        p = nullptr;
    };
    keep(c->spare[0], s.pr64, s.pr_bytes[0]);
    keep(c->spare[1], s.pr32, s.pr_bytes[1]);
    keep(c->spare[2], s.tc_mem[0], s.tc_bytes[0]);
    keep(c->spare[3], s.tc_mem[1], s.tc_bytes[1]);
    unsigned char* mem = s.mem;
    const size_t cap = s.mem_cap;
    s.mem = nullptr;
    slot_free(s);
    s.mem = mem;
    s.mem_cap = cap;
}

// *p = a buffer of at least bytes: the spare when it fits, else a new one
template <typename T>
inline cudaError_t spare_alloc(hpsi_ctx* c, Spare& spare, T** p, size_t* bytes)
{
    if (spare.p && spare.bytes >= *bytes && spare.bytes / 2 <= *bytes) {
        *p = static_cast<T*>(spare.p);
        *bytes = spare.bytes;
        spare = Spare{};
        return cudaSuccess;
    }
    dfree(spare.p);
    spare = Spare{};
    return dev_malloc(c, p, *bytes);
}

inline int ws_reserve(hpsi_ctx* c, size_t bytes)
{
    c->d64_ws = nullptr;
    if (bytes <= c->ws_size) return HPSI_OK;
    if (c->ws != c->ws_first) cudaFree(c->ws);
    c->ws = c->ws_first;
    c->ws_size = c->ws_first_size;
    const size_t want = bytes + bytes / 8;
    unsigned char* p = nullptr;
    CUDA_TRY(c, dev_malloc(c, &p, want));
    c->ws = p;
    c->ws_size = want;
    if (!c->ws_first) {
        c->ws_first = p;
        c->ws_first_size = want;
    }
    return HPSI_OK;
}

// d64_mem of at least bytes; false when the device has no room, or under capture
// (an allocation would end it)
inline bool d64_reserve(hpsi_ctx* c, size_t bytes, cudaStream_t st)
{
    if (bytes <= c->d64_cap) return true;
    if (capturing(st)) return false;
    size_t free_bytes = 0, total = 0;
    if (bytes >= c->d64_refused &&
        (cudaMemGetInfo(&free_bytes, &total) != cudaSuccess || free_bytes <= c->d64_refused_free))
        return false;
    release_optional(c);
    ++c->d64_tries;
    for (size_t want : {bytes + bytes / 8, bytes}) {
        if (want <= c->test_d64_room && cudaMalloc((void**)&c->d64_mem, want) == cudaSuccess) {
            c->d64_cap = want;
            c->d64_refused = SIZE_MAX;
            return true;
        }
        cudaGetLastError();  // not an error of the call
    }
    c->d64_mem = nullptr;
    c->d64_refused = bytes;
    if (cudaMemGetInfo(&c->d64_refused_free, &total) != cudaSuccess) c->d64_refused_free = 0;
    return false;
}

// Reserve base bytes, and extra bytes for the FP64 GEMMs on the tensor cores
// (d64_ws).  Without room for extra the call goes on with base alone.  A workspace
// that has to grow takes a small extra along (one allocation instead of two on the
// first call of a cell: 460 -> 410 us for 8 atoms, 48 bands).
constexpr size_t kExtraInWs = 32u << 20;
inline int ws_reserve_d64(hpsi_ctx* c, size_t base, size_t extra, cudaStream_t st)
{
    const size_t off = (base + 255) / 256 * 256;
    const std::string err = c->err;
    int rc = ws_reserve(c, base > c->ws_size && extra <= std::min(kExtraInWs, c->test_d64_room) ? off + extra : base);
    if (rc == HPSI_ERR_OOM) {
        cudaGetLastError();  // not an error of the call if base alone fits
        c->err = err;
        rc = ws_reserve(c, base);
    }
    if (rc || extra == 0) return rc;
    if (off + extra <= c->ws_size && extra <= c->test_d64_room) {
        c->d64_ws = c->ws + off;
    } else {
        if (!d64_reserve(c, extra, st)) return HPSI_OK;
        c->d64_ws = c->d64_mem;
    }
    c->d64_size = extra;
    return HPSI_OK;
}

// Build, once, what a precision needs on slot s (projector matrices, tensor-core
// operands; with grad also the derivative operands).  Allocates.
int prepare_slot(hpsi_ctx* c, KSlot& s, int prec, bool grad, cudaStream_t st);
