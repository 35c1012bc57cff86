// capi.cu -- the C ABI of include/titan_gb300.h.
//
// Replaces the reference's device-state layer and run loop
// (src/sim.cu:821-1017 AoS per-object cudaMalloc + pointer arrays, and
// src/sim.cu:1503-1617 sync + two launches per step) with: one tile plan,
// structure-of-arrays buffers allocated once, and CUDA-graph replay of the
// fused step kernel on a private stream.
#include "titan_gb300.h"

#include <cuda.h>

#include <algorithm>
#include <array>
#include <cmath>
#include <chrono>
#include <cstring>
#include <thread>
#include <map>
#include <memory>
#include <new>
#include <string>
#include <utility>
#include <vector>

#include "engine.h"
#include "plan.h"

using tg::P_FP32;
using tg::P_FP32C;
using tg::P_FP64;

namespace {

constexpr int kChunk = 64;  // steps per cached graph

double norm3(const double *v) {
    double a = v[0] * v[0], b = v[1] * v[1], c = v[2] * v[2];
    return std::sqrt((a + b) + c);
}

struct DevMem {
    std::vector<void *> ptrs;
    size_t total = 0;
    void *get(size_t bytes, cudaError_t &e) {
        void *p = nullptr;
        if (bytes == 0) bytes = 16;
        e = cudaMalloc(&p, bytes);
        if (e == cudaSuccess) {
            ptrs.push_back(p);
            total += bytes;
        }
        return p;
    }
    void release() {
        for (void *p : ptrs) cudaFree(p);
        ptrs.clear();
        total = 0;
    }
};

}  // namespace

constexpr int kRtGroups = 3;  // size groups of resident tiles

struct titan_gb300_sim {
    int device = 0, prec = P_FP64;
    cudaStream_t stream = nullptr;
    // resident tiles run on side streams beside the per-step kernels
    cudaStream_t side_stream[kRtGroups] = {};
    cudaEvent_t ev_fork = nullptr, ev_join[kRtGroups] = {};
    std::string err;

    // host scene (creation order)
    int64_t n = 0;
    std::vector<double> pos, vel, m, ext, drag_in;
    std::vector<uint8_t> fixed;
    std::vector<int32_t> drag;
    std::vector<int64_t> lc_ptr;  // n+1 or empty
    std::vector<int32_t> lc_type;
    std::vector<double> lc_rec;   // 4 per record
    int64_t ns = 0;
    std::vector<int32_t> left, right, type;
    std::vector<double> k, rest, damping, omega, amp, phase;
    std::vector<std::array<double, 6>> planes;
    std::vector<std::array<double, 4>> balls;
    std::vector<int64_t> body_ptr;
    std::vector<std::array<double, 6>> body_plane;
    std::vector<uint8_t> body_has_plane;
    double dt = 1e-4;
    double g[3] = {0.0, 0.0, -9.81};

    // run state
    bool started = false;
    double T = 0.0;
    int64_t steps = 0;
    int parity = 0;
    std::vector<double> mT0;       // per-mass local time at its last upload
    std::vector<int64_t> mTstep;   // step count at that upload
    struct DtSeg {
        int64_t first;  // first step of the segment
        double dt;
        int halves;     // 2: RK2 advances time by dt/2 twice per step
    };
    std::vector<DtSeg> dt_log;
    int integrator = tg::INTEG_EULER;
    int passes() const { return integrator == tg::INTEG_RK2 ? 2 : 1; }

    // device
    tg::Plan plan;
    DevMem mem;
    tg::StepArgs args{};
    tg::DevParams hprm{};
    tg::DevParams *dprm = nullptr;
    int threads = 512;
    int tile_masses = 0;
    size_t smem = 0;
    int64_t npad = 0;
    int32_t *d_old2new = nullptr;
    double *d_xfer = nullptr;     // 9n doubles
    int64_t *d_idx = nullptr;     // n
    double *h_xfer = nullptr;     // pinned 9n doubles, then the error flag k_gather copies
    double *stage_dev = nullptr;  // h_xfer's address on the device
    int *h_err = nullptr;
    std::map<std::pair<int, int>, cudaGraphExec_t> graphs;
    // diagnostics (lazy)
    int32_t *d_sl = nullptr, *d_sr = nullptr;
    double *d_partials = nullptr, *d_dout = nullptr;
    // spring parameters on the device in creation order (k, rest, damping,
    // omega, amp, phase), each there once something needs it; sp_current: it
    // holds the host array's values.  d_espring: the spring of each slab entry.
    enum { SP_K, SP_REST, SP_DAMPING, SP_OMEGA, SP_AMP, SP_PHASE, SP_COUNT };
    double *d_sp[SP_COUNT] = {};
    bool sp_current[SP_COUNT] = {};
    int32_t *d_espring = nullptr;
    int64_t wait_polls = 0;  // of one halo wait in the resident grid (0: the default)
    // a step kernel gave up a wait: steps are refused until all positions and
    // velocities are uploaded again
    bool torn = false;
    // a kernel that writes the slab records may still run: the next step
    // kernel, which reads them before its grid_dep_wait(), must not start early
    bool tables_written = false;

    size_t rsize() const { return prec == P_FP64 ? sizeof(double) : sizeof(float); }
    int comps() const { return tg::state_words(prec); }
    int threads_req = 0;  // CTA size override (0: derived from the tile size)
    int min_ctas_req = 0; // register cap of the per-tile kernel: 0/1 none, 3 or 4 CTAs per SM
    int step_variant = 0; // launch-bound variant in use (engine.h)
    int kernel_req = 0;   // 0 auto, 1 per-tile kernel, 3 per-tile with async staging, 4 warp-specialised, 6 pull
    bool use_async = false;
    bool use_ws = false;
    bool serving = false;  // handed to a request server (server.cu)
    bool use_pull = false;
    tg::PullTables pull;  // host copy of the pull form's spring tables
    std::vector<tg::PullTile> pull_tiles;
    int64_t pull_impl_bytes = 0;
    int ws_warps = 0;     // consumer warps of the warp-specialised kernel
    int ctas = 0;         // persistent grid of the pipelined kernel
    int *d_err = nullptr;
    // body-resident batched launch
    int res_mode = -1;    // -1 automatic, 0 off, 1 bins of whole bodies, 2 halo-free tiles
    int res_bin_req = 0;  // bin capacity in masses (0: default)
    int res_threads_req = 0;
    tg::ResPlan rplan;
    tg::ResArgs rargs{};
    bool use_res = false;
    int res_threads = 0, res_ctas = 0;
    // resident tiles (mode 2): halo-free tiles stepped in shared memory
    bool use_rtiles = false;
    std::vector<tg::TileInfo> rtiles;
    struct RtGroup {  // a launch's share of them, with its shape
        size_t first = 0;
        tg::TileResArgs args{};
        int threads = 0, mpt = 0;
        size_t smem = 0;
    };
    std::vector<RtGroup> rt_groups;
    // calls of a few steps on scenes with whole bodies above the per-step
    // tile size (short_limit): those bodies in pieces of that size.  The
    // tables are the plan's and behind them the pieces'.
    struct ShortForm {
        bool tried = false, ready = false;
        int64_t calls = 0;  // such calls before the tables were made
        tg::StepArgs args{};
        tg::RepeatArgs pieces{};
        int ctas = 0;
    } short_form;
    double *d_t0 = nullptr;  // the first step's T, where per-step kernels advance the record beside them
    // all tiles at once (resident_grid.cu); the per-step kernels stay ready
    // for single steps
    bool use_grid = false;
    tg::GridResArgs gargs{};
    int grid_shape = 0, single_shape = -1;  // single steps as one pass of it, -1: by the per-step kernels
    size_t grid_smem = 0;
    int grid_last = 0;  // the last step(): 1 resident grid, 2 its single pass, 3 short_form, 0 other kernels
    // plan taken from another handle with the same topology (adopt_plan);
    // used by the first start() only
    bool plan_adopted = false;
    int plan_tile = 0;  // tile size the current plan was built with
    int plan_req = 0;   // tile size requested for it (0: the default)
    // sizes that the handle's settings asked the planner for: tile, smallest
    // tile, whole bodies, cut
    std::array<int, 4> plan_ask{};

    cudaError_t launch(int parity, int write_acc, int stage = 0) {
        if (args.ntiles == 0) return cudaSuccess;
        args.rk2_stage = stage;
        if (use_pull) return tg::launch_step_pull(prec, integrator, args, ctas, parity, write_acc, stream);
        if (use_ws)
            return tg::launch_step_ws(prec, integrator, args, ctas, ws_warps, parity, write_acc, stream, !tables_written);
        if (use_async)
            return tg::launch_step_async(prec, args, (int)args.ntiles, threads, smem, parity, write_acc, stream);
        return tg::launch_step(prec, step_variant, integrator, args, (int)args.ntiles, threads, smem, parity,
                               write_acc, stream);
    }

    int fail(int code, const std::string &msg) {
        err = msg;
        return code;
    }
    int cuda_fail(cudaError_t e, const char *what) {
        err = std::string(what) + ": " + cudaGetErrorString(e);
        return TITAN_GB300_ECUDA;
    }

    void drop_graphs() {
        for (auto &kv : graphs) cudaGraphExecDestroy(kv.second);
        graphs.clear();
    }
    void free_device() {
        drop_graphs();
        mem.release();
        if (h_xfer) cudaFreeHost(h_xfer);
        h_xfer = nullptr;
        h_err = nullptr;
        d_sl = d_sr = nullptr;
        d_partials = d_dout = nullptr;
        for (int q = 0; q < SP_COUNT; q++) d_sp[q] = nullptr, sp_current[q] = false;
        d_espring = nullptr;
        short_form = ShortForm{};
    }
    ~titan_gb300_sim() {
        if (stream) cudaStreamSynchronize(stream);
        free_device();
        if (stream) cudaStreamDestroy(stream);
        for (cudaStream_t st : side_stream) {
            if (!st) continue;
            cudaStreamSynchronize(st);
            cudaStreamDestroy(st);
        }
        if (ev_fork) cudaEventDestroy(ev_fork);
        for (cudaEvent_t ev : ev_join)
            if (ev) cudaEventDestroy(ev);
    }
};

namespace {

#define CK(call, what)                                  \
    do {                                                \
        cudaError_t e_ = (call);                        \
        if (e_ != cudaSuccess) return s->cuda_fail(e_, what); \
    } while (0)

// A host buffer's address on the device where all its bytes lie in one
// page-locked range (cudaMallocHost or cudaHostRegister) that the device may
// write, null for other memory: kernels store there, and a store past the
// range (an array registered in part) or into a read-only registration would
// be an illegal access.
void *host_on_device(const void *p, size_t bytes) {
    cudaPointerAttributes at{};
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    if (at.type != cudaMemoryTypeHost || !at.devicePointer) return nullptr;
    using Query = CUresult (*)(void *, CUpointer_attribute, CUdeviceptr);
    static const Query query = [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult found{};
        if (cudaGetDriverEntryPointByVersion("cuPointerGetAttribute", &f, 12000, cudaEnableDefault, &found) != cudaSuccess) {
            cudaGetLastError();
            f = nullptr;
        }
        return reinterpret_cast<Query>(found == cudaDriverEntryPointSuccess ? f : nullptr);
    }();
    const CUdeviceptr d = (CUdeviceptr)at.devicePointer;
    CUdeviceptr start = 0;
    size_t size = 0;
    int access = 0;
    if (!query || query(&start, CU_POINTER_ATTRIBUTE_RANGE_START_ADDR, d) != CUDA_SUCCESS ||
        query(&size, CU_POINTER_ATTRIBUTE_RANGE_SIZE, d) != CUDA_SUCCESS ||
        query(&access, CU_POINTER_ATTRIBUTE_ACCESS_FLAGS, d) != CUDA_SUCCESS)
        return nullptr;
    const bool inside = d >= start && bytes <= size && d - start <= size - bytes;
    return inside && access == CU_POINTER_ATTRIBUTE_ACCESS_FLAG_READWRITE ? at.devicePointer : nullptr;
}

// Whether a caller's host buffer is page-locked (cudaMallocHost or
// cudaHostRegister): such buffers are copied by DMA directly, without the
// staging copy through the handle's own pinned buffer.
bool host_pinned(const void *p) {
    if (!p) return false;
    cudaPointerAttributes at{};
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
        cudaGetLastError();  // clear the error state the failed query left
        return false;
    }
    return at.type == cudaMemoryTypeHost;
}

// memcpy of large host buffers split over a few threads (the staging copies
// of whole-scene state are tens of MB; one core copies them at a fraction of
// the host memory bandwidth, and a new destination's pages are first touched
// here: 15 MB of velocities into a new array took 1.39 ms with pieces of 8 MB).
void par_memcpy(void *dst, const void *src, size_t bytes) {
    constexpr size_t kPiece = 2u << 20;
    // (asked once: the answer takes 6 us)
    static const unsigned hw = std::max(1u, std::thread::hardware_concurrency());
    const size_t nt = std::min<size_t>(std::min<size_t>(8, hw), (bytes + kPiece - 1) / kPiece);
    if (nt <= 1) {
        std::memcpy(dst, src, bytes);
        return;
    }
    const size_t per = (bytes / nt + 63) & ~size_t(63);
    std::vector<std::thread> th;
    for (size_t q = 1; q < nt; q++) {
        const size_t o = q * per;
        if (o >= bytes) break;
        th.emplace_back([=] {
            std::memcpy(static_cast<uint8_t *>(dst) + o, static_cast<const uint8_t *>(src) + o, std::min(per, bytes - o));
        });
    }
    std::memcpy(dst, src, std::min(per, bytes));
    for (auto &t : th) t.join();
}

uint8_t mass_flags(const titan_gb300_sim *s, int64_t i) {
    uint8_t f = 0;
    if (!s->fixed.empty() && s->fixed[i]) f |= tg::MF_FIXED;
    if (!s->ext.empty() && (s->ext[3 * i] != 0.0 || s->ext[3 * i + 1] != 0.0 || s->ext[3 * i + 2] != 0.0))
        f |= tg::MF_EXT;
    if (!s->drag.empty() && s->drag[i] != 0) f |= tg::MF_DRAG;
    if (!s->lc_ptr.empty() && s->lc_ptr[i + 1] > s->lc_ptr[i]) f |= tg::MF_LOCAL;
    return f;
}

void fill_params(titan_gb300_sim *s) {
    tg::DevParams &p = s->hprm;
    std::memset(&p, 0, sizeof(p));
    p.dt = s->dt;
    p.dt_hi = (float)s->dt;
    p.dt_lo = (float)(s->dt - (double)p.dt_hi);
    p.integrator = s->integrator;
    p.dt2 = std::pow(s->dt, 2);
    p.dt2f = (float)p.dt2;
    p.launch_dt = s->integrator == tg::INTEG_RK2 ? 0.5 * s->dt : s->dt;
    for (int c = 0; c < 3; c++) {
        p.g[c] = s->g[c];
        p.gf[c] = (float)s->g[c];
    }
    p.nplanes = (int32_t)s->planes.size();
    p.nballs = (int32_t)s->balls.size();
    for (size_t j = 0; j < s->planes.size(); j++)
        for (int c = 0; c < 6; c++) {
            p.plane[j][c] = s->planes[j][c];
            p.planef[j][c] = (float)s->planes[j][c];
        }
    for (size_t j = 0; j < s->balls.size(); j++)
        for (int c = 0; c < 4; c++) {
            p.ball[j][c] = s->balls[j][c];
            p.ballf[j][c] = (float)s->balls[j][c];
        }
}

int upload_params(titan_gb300_sim *s) {
    fill_params(s);
    CK(cudaMemcpyAsync(s->dprm, &s->hprm, sizeof(tg::DevParams), cudaMemcpyHostToDevice, s->stream),
       "upload params");
    CK(cudaMemcpyAsync(s->args.tbuf + s->parity, &s->T, sizeof(double), cudaMemcpyHostToDevice, s->stream),
       "upload time");
    CK(cudaStreamSynchronize(s->stream), "upload params");
    return TITAN_GB300_OK;
}

template <typename R>
std::vector<R> to_real(const std::vector<double> &v) {
    return std::vector<R>(v.begin(), v.end());
}

// Per-mass device arrays (m, flags, ext, drag, local constraints) from the
// host mirror, in tiled order.
int upload_mass_attrs(titan_gb300_sim *s) {
    const tg::Plan &P = s->plan;
    const int64_t n = s->n, np = s->npad;
    std::vector<uint8_t> flags(np, tg::MF_FIXED);
    std::vector<double> md(np, 1.0), extd(3 * np, 0.0);
    std::vector<int32_t> dragn(np, 0), lcp(np + 1, 0);
    std::vector<int32_t> lct;
    std::vector<double> lcr;
    for (int64_t g = 0; g < n; g++) {
        int64_t i = P.new2old[g];
        uint8_t f = mass_flags(s, i);
        int32_t b = 0;
        if (!s->body_ptr.empty())
            b = (int32_t)(std::upper_bound(s->body_ptr.begin(), s->body_ptr.end(), i) - s->body_ptr.begin() - 1);
        if (!s->body_has_plane.empty() && s->body_has_plane[b]) f |= tg::MF_BODYPLANE;
        flags[g] = f;
        md[g] = s->m[i];
        if (!s->ext.empty())
            for (int c = 0; c < 3; c++) extd[c * np + g] = s->ext[3 * i + c];
        if (!s->drag.empty()) dragn[g] = s->drag[i];
        lcp[g] = (int32_t)lct.size();
        if (!s->lc_ptr.empty())
            for (int64_t r = s->lc_ptr[i]; r < s->lc_ptr[i + 1]; r++) {
                lct.push_back(s->lc_type[r]);
                for (int c = 0; c < 4; c++) lcr.push_back(s->lc_rec[4 * r + c]);
            }
    }
    for (int64_t g = n; g <= np; g++) lcp[g] = (int32_t)lct.size();
    auto &a = s->args;
    CK(cudaMemcpy(const_cast<uint8_t *>(a.flags), flags.data(), np, cudaMemcpyHostToDevice), "upload flags");
    if (s->prec == P_FP64) {
        CK(cudaMemcpy(const_cast<void *>(a.mass), md.data(), np * 8, cudaMemcpyHostToDevice), "upload m");
        CK(cudaMemcpy(const_cast<void *>(a.ext), extd.data(), 3 * np * 8, cudaMemcpyHostToDevice), "upload ext");
    } else {
        auto mf = to_real<float>(md);
        auto ef = to_real<float>(extd);
        CK(cudaMemcpy(const_cast<void *>(a.mass), mf.data(), np * 4, cudaMemcpyHostToDevice), "upload m");
        CK(cudaMemcpy(const_cast<void *>(a.ext), ef.data(), 3 * np * 4, cudaMemcpyHostToDevice), "upload ext");
    }
    CK(cudaMemcpy(const_cast<int32_t *>(a.drag), dragn.data(), np * 4, cudaMemcpyHostToDevice), "upload drag");
    CK(cudaMemcpy(const_cast<int32_t *>(a.lc_ptr), lcp.data(), (np + 1) * 4, cudaMemcpyHostToDevice), "upload lc");
    if (!lct.empty()) {
        cudaError_t e;
        int32_t *t = (int32_t *)s->mem.get(lct.size() * 4, e);
        if (!t) return s->cuda_fail(e, "alloc lc");
        double *r = (double *)s->mem.get(lcr.size() * 8, e);
        if (!r) return s->cuda_fail(e, "alloc lc");
        CK(cudaMemcpy(t, lct.data(), lct.size() * 4, cudaMemcpyHostToDevice), "upload lc");
        CK(cudaMemcpy(r, lcr.data(), lcr.size() * 8, cudaMemcpyHostToDevice), "upload lc");
        a.lc_type = t;
        a.lc_rec = r;
    }
    return TITAN_GB300_OK;
}

tg::PullSprings pull_springs(const titan_gb300_sim *s) {
    tg::PullSprings sp;
    sp.k = s->k.data();
    sp.rest = s->rest.data();
    sp.damping = s->damping.empty() ? nullptr : s->damping.data();
    return sp;
}

// Spring records (slab-entry layout: FP64 k, rest, damping, word; FP32
// word, k, rest, damping) and actuation records for the springs spring[e]
// with entry words word[e] (spring -1: a zero padding record), uploaded to
// rec / act.
int upload_records(titan_gb300_sim *s, const std::vector<int64_t> &spring, const std::vector<uint32_t> &word,
                   void *rec, void *act) {
    const size_t E = spring.size();
    if (E == 0) return TITAN_GB300_OK;
    auto sp_amp = [&](int64_t j) { return s->amp.empty() ? 0.2 : s->amp[j]; };
    auto sp_phase = [&](int64_t j) { return s->phase.empty() ? 0.0 : s->phase[j]; };
    auto sp_omega = [&](int64_t j) { return s->omega.empty() ? 0.0 : s->omega[j]; };
    if (s->prec == P_FP64) {
        std::vector<double> ent(4 * E, 0.0), ac(4 * E, 0.0);
        for (size_t e = 0; e < E; e++) {
            int64_t j = spring[e];
            if (j < 0) continue;
            ent[4 * e] = s->k[j];
            ent[4 * e + 1] = s->rest[j];
            ent[4 * e + 2] = s->damping[j];
            uint64_t bits = word[e];
            std::memcpy(&ent[4 * e + 3], &bits, 8);
            ac[4 * e] = sp_omega(j);
            ac[4 * e + 1] = sp_amp(j);
            ac[4 * e + 2] = sp_phase(j);
        }
        CK(cudaMemcpy(rec, ent.data(), ent.size() * 8, cudaMemcpyHostToDevice), "upload records");
        CK(cudaMemcpy(act, ac.data(), ac.size() * 8, cudaMemcpyHostToDevice), "upload actuation");
    } else {
        std::vector<float> ent(4 * E, 0.f), ac(4 * E, 0.f);
        for (size_t e = 0; e < E; e++) {
            int64_t j = spring[e];
            if (j < 0) continue;
            uint32_t bits = word[e];
            std::memcpy(&ent[4 * e], &bits, 4);
            ent[4 * e + 1] = (float)s->k[j];
            ent[4 * e + 2] = (float)s->rest[j];
            ent[4 * e + 3] = (float)s->damping[j];
            // rest' = rest (1 + a sin(2 pi (nu T + phi))): nu = omega / 2 pi,
            // phi = phase / 2 pi, a = -amp for contract-then-expand (type 2)
            const double two_pi = 6.283185307179586476925286766559;
            const int ty = s->type.empty() ? 0 : s->type[j];
            ac[4 * e] = (float)(sp_omega(j) / two_pi);
            ac[4 * e + 1] = (float)(ty == 2 ? -sp_amp(j) : sp_amp(j));
            ac[4 * e + 2] = (float)(sp_phase(j) / two_pi);
            ac[4 * e + 3] = (float)s->rest[j];  // read by the pull form with the record
        }
        CK(cudaMemcpy(rec, ent.data(), ent.size() * 4, cudaMemcpyHostToDevice), "upload records");
        CK(cudaMemcpy(act, ac.data(), ac.size() * 4, cudaMemcpyHostToDevice), "upload actuation");
    }
    return TITAN_GB300_OK;
}

// The records of the tables for calls of a few steps, from the plan's.
int refresh_short(titan_gb300_sim *s) {
    const auto &f = s->short_form;
    const size_t bytes = s->plan.ent_ends.size() * (size_t)tg::entry_record_bytes(s->prec);
    CK(cudaMemcpyAsync(const_cast<void *>(f.args.ent), s->args.ent, bytes, cudaMemcpyDeviceToDevice, s->stream), "copy records");
    CK(cudaMemcpyAsync(const_cast<void *>(f.args.act), s->args.act, bytes, cudaMemcpyDeviceToDevice, s->stream), "copy records");
    CK(tg::launch_repeat_entries(s->prec, f.pieces, s->stream), "repeat records");
    s->tables_written = true;
    return TITAN_GB300_OK;
}

// Slab entry records and actuation parameters from the host spring arrays,
// and the resident bins' records.
int upload_entries(titan_gb300_sim *s) {
    const tg::Plan &P = s->plan;
    auto &a = s->args;
    int rc = upload_records(s, P.ent_spring, P.ent_ends, const_cast<void *>(a.ent), const_cast<void *>(a.act));
    if (rc) return rc;
    if (s->use_pull && a.pull_units) {  // new spring parameters: same layout, new values
        tg::PullTables T;
        std::string why = tg::build_pull(P, s->pull_tiles, s->pull.team_warps, tg::state_record_bytes(s->prec) / 16,
                                         pull_springs(s), T);
        if (!why.empty()) return s->fail(TITAN_GB300_ELIMIT, why);
        if (T.units.size() != s->pull.units.size() || T.ell.size() != s->pull.ell.size())
            return s->fail(TITAN_GB300_EINVAL, "pull tables changed shape without a new plan");
        s->pull = std::move(T);
        CK(cudaMemcpy(const_cast<tg::PullUnit *>(a.pull_units), s->pull.units.data(),
                      s->pull.units.size() * sizeof(tg::PullUnit), cudaMemcpyHostToDevice),
           "upload pull units");
        CK(cudaMemcpy(const_cast<uint8_t *>(a.pull_ell), s->pull.ell.data(), s->pull.ell.size(),
                      cudaMemcpyHostToDevice),
           "upload pull columns");
    }
    if (s->short_form.ready)
        if (int rs = refresh_short(s)) return rs;
    if (s->use_res)
        rc = upload_records(s, s->rplan.rec_spring, s->rplan.words, const_cast<void *>(s->rargs.rec),
                            const_cast<void *>(s->rargs.act));
    return rc;
}

template <typename T>
T *dev_copy(titan_gb300_sim *s, const std::vector<T> &v, cudaError_t &e) {
    T *p = (T *)s->mem.get(v.size() * sizeof(T), e);
    if (!p) return nullptr;
    if (!v.empty()) e = cudaMemcpy(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice);
    return e == cudaSuccess ? p : nullptr;
}

// default tile of the warp-specialised form, and its fallback when two
// stages of the default's tiles do not fit one SM's shared memory
constexpr int kWsDefaultTile = 208;
constexpr int kWsFallbackTile = 192;
// default tile of the pull form: seven 32-mass units, one per warp of a team
// (two teams and the producer: 16 warps, four per SM sub-partition)
constexpr int kPullDefaultTile = 224;
// the automatic kernel choice in FP32 and FP32C: the warp-specialised form
// (measured faster on GB300 on the 100^3 lattice: 0.121 ms per step against
// 0.134 for the pull form with 160-mass tiles and three teams)
constexpr bool kPullAuto = false;
constexpr int kHeavyThreshold = 96;
constexpr int64_t kGridMinSteps = 2;
// Single steps of a scene planned for the resident grid run as one pass of
// its kernel up to this many masses a tile (26^3: 5.9 us against 6.5 with
// the warp-specialised kernel; 30^3, 89 masses a tile: 7.8 against 7.0), with
// 256 threads a CTA (12^3: 4.0 us against 4.4 with 128).
constexpr int kSingleMasses = 64, kSingleShape = 1;

// Steps of one resident-grid launch: other handles' kernels get no SM that its
// CTAs fill until it ends, so long calls are cut (100 steps of a 24^3 scene
// beside 200,000 of a 9^3 one, FP64: 5 ms; in one launch 1.39 s, to that one's
// end).  A launch costs about 6 us more than its steps, 0.1 to 0.4 % of 512.
constexpr int64_t kGridMaxSteps = 512;

// Whether the step will run the pull form: when requested (set_kernel 6).
// (It needs a plan without heavy masses: it has no warp-cooperative sums.)
bool pull_wanted(const titan_gb300_sim *s) {
    if (s->kernel_req == 6) return true;
    if (!kPullAuto || s->kernel_req != 0 || s->prec == P_FP64) return false;
    std::vector<int32_t> deg(s->n, 0);
    for (int64_t j = 0; j < s->ns; j++) {
        const int64_t l = s->left[j], r = s->right[j];
        if (l < 0 || r < 0 || l >= s->n || r >= s->n) continue;
        if (++deg[l] > kHeavyThreshold && (s->fixed.empty() || !s->fixed[l])) return false;
        if (++deg[r] > kHeavyThreshold && (s->fixed.empty() || !s->fixed[r])) return false;
    }
    return true;
}

int sm_count(const titan_gb300_sim *s) {
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s->device) != cudaSuccess || sms <= 0) {
        cudaGetLastError();
        sms = 152;  // GB300
    }
    return sms;
}

std::array<int, 4> plan_sizes(const tg::PlanInput &in) { return {in.tile_cap, in.tile_min, in.whole_cap, in.cut_above}; }

// Whether nothing chose another form than the resident grid for calls of
// several steps.
bool grid_wanted(const titan_gb300_sim *s) {
    return s->kernel_req == 0 && s->res_mode == -1 && s->threads_req == 0 && s->min_ctas_req == 0 &&
           s->res_threads_req == 0;
}

// The resident grid's launch for these tiles (resident_grid.cu): every tile
// gets a CTA at once, with the slab in shared memory if that fits.  Small
// tiles get small CTAs, which leave the SMs to other handles' kernels: FP64
// 256 threads up to 600 entries, else 512.  From 300 to 600 entries (2,000 to
// 4,500 masses) the wider CTA is 10 % faster alone (14^3: 7.4 us per step
// against 8.2; a 61 x 11 x 7 beam with drag and a ball 5 %; above, 17^3: 9.6
// against 10.4), but it fills the SM, so that
// scenes in flight together take turns: 4 scenes of 27 to 4,000 masses, 300
// steps, 6.2 against 3.0 ms, 24 of 27 to 3,000, 190 steps, 12.8 against 9.8.
// 128 threads: 9^3 7.5 us against 6.2.  The FP32 forms 128 up to 400 entries,
// else 256 (16^3: 2.85 us with 128, 3.1 with 256; 24 scenes of 27 to 60,000
// masses in flight together, 200 steps: 8.2 against 10.5 ms).  128 threads in
// FP64 and 512 in the FP32 forms are taken where the others refuse, which
// with the default sizes they do not: tiles asked for by start() of more than
// 256 masses (FP32), or of more than 304 in number (FP64).  Returns false when
// the tiles do not all fit.
bool choose_grid(const titan_gb300_sim *s, const std::vector<tg::TileInfo> &tiles, int &shape, int &stage, size_t &bytes) {
    size_t smem[2] = {0, 0};
    int max_nm = 0, max_ne = 0;
    for (const tg::TileInfo &ti : tiles) {
        max_nm = std::max(max_nm, (int)ti.nm);
        max_ne = std::max(max_ne, (int)ti.ne);
        for (int st = 0; st < 2; st++) smem[st] = std::max(smem[st], tg::grid_resident_smem_bytes(s->prec, ti, st));
    }
    int first;
    if (s->prec == P_FP64) first = max_ne <= 600 ? 1 : 0;
    else first = max_ne <= 400 ? 2 : 1;
    const int order[3][tg::kGridShapes] = {{0, 1, 2}, {1, 0, 2}, {2, 1, 0}};
    for (const int sh : order[first]) {
        shape = sh;
        const int ctas = tg::grid_resident_ctas(shape);
        if ((int64_t)tiles.size() > (int64_t)sm_count(s) * ctas || max_nm > tg::grid_resident_threads(shape))
            continue;
        for (stage = 1; stage >= 0; stage--)
            if (smem[stage] <= 227 * 1024 && (smem[stage] + 1024) * ctas <= 228 * 1024) {
                bytes = smem[stage];
                return true;
            }
    }
    return false;
}

// Tile size with which the resident grid has all tiles at once, 0 if none:
// the smallest that leaves one tile per SM in FP64 (each SM's FP64 pipe and
// issue slots bind, and one CTA then has 512 threads) and two in the FP32
// forms, where two CTAs fill each other's waits.  Measured, us per step, in
// FP64 at 1 and 2 tiles per SM: 24^3 18.0 and 19.0, 30^3 28.9 and 31.0; in
// FP32C 16^3 3.48 and 3.15, 30^3 6.6 and 6.2 -- and with the per-step
// kernels 22.4, 32.2, 4.1 and 7.9 (all before later steps: now 17.4, 28.0,
// 2.7 and 5.7 with the sizes chosen here).  At least 8 masses per tile in FP64 (9^3:
// 7.4 us per step against 8.0 with 16), 16 in the FP32 forms (2.7 against 2.5
// with 8, but half the CTAs).  Bodies up to whole masses stay one tile.
// Above 192 masses (FP64) or 208 (FP32C: 63,000 in all) per tile the SM's
// shared memory is too small; FP64 batches of bodies then try two per SM.
int grid_tile(const titan_gb300_sim *s, int whole) {
    const int64_t sms = sm_count(s);
    auto tiles_of = [&](int t) {
        if (s->body_ptr.empty()) return s->n <= whole ? (int64_t)1 : (s->n + t - 1) / t;
        int64_t k = 0;
        for (size_t b = 0; b + 1 < s->body_ptr.size(); b++) {
            const int64_t m = s->body_ptr[b + 1] - s->body_ptr[b];
            k += m <= whole ? 1 : (m + t - 1) / t;
        }
        return k;
    };
    auto smallest = [&](int64_t most, int hi) {
        if (tiles_of(hi) > most) return 0;
        int lo = std::min(hi, s->prec == P_FP64 ? 8 : 16);
        while (lo < hi) {
            const int mid = (lo + hi) / 2;
            if (tiles_of(mid) <= most) hi = mid;
            else lo = mid + 1;
        }
        return hi;
    };
    if (s->prec != P_FP64) return smallest(2 * sms, kWsDefaultTile);
    const int t = smallest(sms, 192);
    return t ? t : smallest(2 * sms, 128);
}

// grid: tiles for the resident grid where grid_tile has a size
tg::PlanInput plan_input(titan_gb300_sim *s, int tile_masses, bool grid = false) {
    tg::PlanInput in;
    in.n = s->n;
    in.pos = s->pos.data();
    in.fixed = s->fixed.empty() ? nullptr : s->fixed.data();
    in.ns = s->ns;
    in.left = s->left.data();
    in.right = s->right.data();
    in.type = s->type.empty() ? nullptr : s->type.data();
    in.nbodies = s->body_ptr.empty() ? 0 : (int64_t)s->body_ptr.size() - 1;
    in.body_ptr = s->body_ptr.empty() ? nullptr : s->body_ptr.data();
    // Default tile.  Large scenes: 96 masses in FP64 (three CTAs per SM,
    // step_var.cu: 80^3 449 us per step against 496 with 256; 256 where a form
    // was chosen), 208 for the FP32 forms' warp-specialised
    // kernel (two stages fit one SM's shared memory; 192 where they would
    // not, plan_scene) and 256 for the per-tile forms.  Smaller scenes get
    // smaller tiles so that their tiles cover the SMs: FP64 about 1.6 tiles
    // per SM (tiles of 32 to 96 masses), the warp-specialised form about
    // 4 (64 to 208).  In the FP32 forms a body that fits the large-scene
    // tile stays whole (a halo-free tile runs resident on one SM: 2.00 us per
    // step for the 5^3 lattice; in the resident grid as eight tiles of 16
    // masses 1.83, as four of 32 2.01); in FP64, bound by each SM's FP64 pipe,
    // it is split like the rest (5^3: 4.6 us in 16 tiles).
    // Measured on GB300, 20^3 lattice, per-step kernels: FP64 16.1 us per
    // step with 32-mass tiles; FP32C 5.3 us with 64 against 6.5 with 208.
    const bool pull = pull_wanted(s);
    const bool ws = !pull && (s->kernel_req == 0 || s->kernel_req == 4);
    if (tile_masses > 0) {
        in.tile_cap = tile_masses;
    } else {
        const int sms = sm_count(s);
        auto fit = [&](double per_sm, int lo, int hi) {
            const int64_t t = (int64_t)((double)s->n / (per_sm * sms)) / 32 * 32;
            return (int)std::max<int64_t>(lo, std::min<int64_t>(hi, t));
        };
        if (s->prec == P_FP64) {
            in.tile_cap = fit(1.6, 32, grid_wanted(s) ? 96 : 256);  // small bodies split too: FP64 binds per SM
        } else if (pull) {
            in.tile_cap = fit(4.0, 64, kPullDefaultTile);
            in.whole_cap = kPullDefaultTile;
        } else if (ws) {
            in.tile_cap = fit(4.0, 64, kWsDefaultTile);
            in.whole_cap = kWsDefaultTile;
            // many bodies: whole ones of up to 512 masses run resident
            // (Euler), a step of 608 bodies of 6^3 masses in 8.9 us against
            // 16.5 as two tiles each, of 8^3 in 24.8 against 30.7; of 9^3 in
            // 42.6 either way.  Calls of a few steps take those bodies in
            // tiles of the size above (short_limit), over the same masses
            if (grid_wanted(s) && s->integrator == tg::INTEG_EULER &&
                (int64_t)s->body_ptr.size() > 2 * (int64_t)sms) {
                in.whole_cap = 512;
                in.cut_above = kWsDefaultTile;
            }
        } else {
            in.tile_cap = 256;
        }
        if (const int t = grid && grid_wanted(s) && !pull ? grid_tile(s, in.whole_cap) : 0) {
            in.tile_cap = t;
            in.tile_min = 8;
        }
    }
    in.heavy_threshold = kHeavyThreshold;
    // a tile's staged state, entry forces and heavy sums share one CTA's
    // shared memory (tile_smem_bytes)
    const int rs = (int)s->rsize();
    in.slot_cap = 4095;
    in.entry_cap = 32767;
    in.smem_budget = 220 * 1024;
    in.slot_bytes = tg::state_record_bytes(s->prec);
    in.entry_bytes = tg::entry_record_bytes(s->prec);
    in.heavy_bytes = 3 * rs;
    return in;
}

// Bin capacity of the resident plan (0: no resident bins): two state
// records per mass must fit one CTA's shared memory, with at most
// kResMaxMpt masses per thread.
int resident_cap(const titan_gb300_sim *s) {
    const int64_t nb = s->body_ptr.empty() ? 1 : (int64_t)s->body_ptr.size() - 1;
    const bool want = s->res_mode == 1;
    if (!want) return 0;
    const int rec = tg::state_record_bytes(s->prec);
    int lim = (int)(((227 * 1024 - 1024) / (2 * rec)) & ~31);
    lim = std::min(lim, tg::kResMaxMpt * (s->res_threads_req > 0 ? s->res_threads_req : 512));
    int64_t big = 0, fit = 0;
    for (int64_t b = 0; b < nb; b++) {
        const int64_t m = s->body_ptr.empty() ? s->n : s->body_ptr[b + 1] - s->body_ptr[b];
        if (m <= lim) big = std::max(big, m), fit++;
    }
    if (big == 0) return 0;
    // default: bins of at least 1024 masses pack small bodies; with no more
    // bodies than one wave of single-body bins (152 SMs), one body per bin
    // of its own size (more CTAs, less shared memory each)
    const int64_t dflt = fit <= 152 ? big : std::max<int64_t>(1024, big);
    const int cap = s->res_bin_req > 0 ? s->res_bin_req : (int)dflt;
    return std::min(lim, (cap + 31) & ~31);
}

// Per-tile launch records of a plan.
std::vector<tg::TileInfo> tile_infos(const tg::Plan &P) {
    std::vector<tg::TileInfo> tiles(P.ntiles);
    for (int64_t t = 0; t < P.ntiles; t++) {
        tg::TileInfo &ti = tiles[t];
        ti.mass_off = (int32_t)P.tile_mass_off[t];
        ti.nm = (int32_t)(P.tile_mass_off[t + 1] - P.tile_mass_off[t]);
        ti.halo_off = (int32_t)P.tile_halo_off[t];
        ti.nh = P.tile_nh[t];
        ti.ent_off = (int32_t)P.tile_ent_off[t];
        ti.ne = (int32_t)(P.tile_ent_off[t + 1] - P.tile_ent_off[t]);
        ti.nact = P.tile_nact[t];
        ti.warp_off = (int32_t)P.tile_warp_off[t];
        ti.heavy_off = (int32_t)P.tile_heavy_off[t];
        ti.nheavy = (int32_t)(P.tile_heavy_off[t + 1] - P.tile_heavy_off[t]);
        ti.body = P.body_of_tile[t];
        const int64_t w0 = P.tile_warp_off[t], w1 = P.tile_warp_off[t + 1];
        const int64_t i0 = w1 > w0 ? (int64_t)P.warp_inc_off[w0] : 0;
        const int64_t i1 = w1 > w0 ? (w1 < (int64_t)P.warp_inc_off.size() ? (int64_t)P.warp_inc_off[w1]
                                                                           : (int64_t)P.inc.size())
                                   : 0;
        ti.inc_off = (int32_t)i0;
        ti.inc_words = (int32_t)(i1 - i0);
        ti.pad0 = ti.pad1 = ti.pad2 = 0;
    }
    return tiles;
}

// Stage layout of the warp-specialised kernel for these tiles (sized by
// their largest): the offsets inside a stage, the halo-index and heavy-sum
// capacities, and how many stages fit one SM's shared memory (nstages; the
// kernel needs at least two).
void ws_stage_layout(int prec, const std::vector<tg::TileInfo> &tiles, tg::WsLayout &W) {
    auto al = [](int64_t x, int64_t q) { return (x + q - 1) / q * q; };
    const int rec = tg::state_record_bytes(prec), ent = tg::entry_record_bytes(prec);
    const int64_t rs = prec == P_FP64 ? 8 : 4;
    int64_t mS = 0, mE = 0, mH = 0, mNh = 0, mA = 0, mI = 0;
    for (const tg::TileInfo &ti : tiles) {
        mS = std::max<int64_t>(mS, ti.nm + ti.nh);
        mE = std::max<int64_t>(mE, ti.ne);
        mH = std::max<int64_t>(mH, ti.nheavy);
        mNh = std::max<int64_t>(mNh, ti.nh);
        mA = std::max<int64_t>(mA, ti.nact);
        mI = std::max<int64_t>(mI, ti.inc_words);
    }
    W.slots = (int32_t)al(mS * rec, 16);
    W.act = (int32_t)al(W.slots + (mE + 1) * ent, 16);  // + the zero slot padding codes name
    W.inc = (int32_t)al(W.act + mA * ent, 16);
    W.stage = (int32_t)al(W.inc + mI * 2, 128);
    W.idx_words = (int32_t)al(mNh, 4);
    W.heavy_cap = (int32_t)std::max<int64_t>(1, mH);
    const int64_t tail = 2 * (int64_t)W.idx_words * 4 + al(2 * 3 * (int64_t)W.heavy_cap * rs, 16) +
                         tg::kWsMaxStages * (int64_t)sizeof(tg::TileInfo) + al((int64_t)sizeof(tg::DevParams), 16) +
                         (2 * tg::kWsMaxStages + 2) * 8 + 32;
    const int64_t room = 227 * 1024 - tail;
    W.nstages = (int32_t)std::min<int64_t>(tg::kWsMaxStages, room / std::max<int64_t>(1, W.stage));
}

// The rest of the layout, behind W.nstages >= 2 stages.
void ws_tail_layout(int prec, tg::WsLayout &W) {
    auto al = [](int64_t x, int64_t q) { return (x + q - 1) / q * q; };
    const int64_t rs = prec == P_FP64 ? 8 : 4;
    W.idx = W.nstages * W.stage;
    W.heavy = W.idx + 2 * W.idx_words * 4;
    W.tinfo = (int32_t)al(W.heavy + 2 * 3 * (int64_t)W.heavy_cap * rs, 16);
    W.params = W.tinfo + W.nstages * (int32_t)sizeof(tg::TileInfo);
    W.mbar = (int32_t)al(W.params + (int64_t)sizeof(tg::DevParams), 16);
    W.total = W.mbar + (2 * W.nstages + 2) * 8 + 32;
}

// Shared-memory layout of the pull kernel for these tiles (sized by their
// largest): stages of one tile's state records, as many as fit one SM (at
// most kPullMaxStages, a multiple of the team count, at least two per
// team).  Returns false when that many do not fit.
bool pull_layout(int prec, const std::vector<tg::TileInfo> &tiles, int threads_req, tg::PullLayout &L) {
    auto al = [](int64_t x, int64_t q) { return (x + q - 1) / q * q; };
    const int rec = tg::state_record_bytes(prec);
    int64_t mS = 0, mNm = 0, mNh = 0, mA = 0;
    for (const tg::TileInfo &ti : tiles) {
        mS = std::max<int64_t>(mS, ti.nm + ti.nh);
        mNm = std::max<int64_t>(mNm, ti.nm);
        mNh = std::max<int64_t>(mNh, ti.nh);
        mA = std::max<int64_t>(mA, ti.nact);
    }
    L = tg::PullLayout{};
    L.team_warps = (int32_t)std::max<int64_t>(1, (mNm + 31) / 32);
    if (L.team_warps > tg::kPullMaxConsumerWarps) return false;
    // two teams by default (one team's narrow tile start and end overlap
    // the other's streaming); set_launch's thread count asks for another
    const int want = threads_req > 0 ? threads_req / 32 / L.team_warps : 2;
    L.nteams = std::max(1, std::min(want, tg::kPullMaxConsumerWarps / L.team_warps));
    L.act_off = (int32_t)al(mS * rec, 16);
    L.stage = (int32_t)al(L.act_off + mA * 16, 128);
    L.idx_words = (int32_t)al(std::max<int64_t>(mNh, 1), 4);
    const int64_t tail = 2 * (int64_t)L.idx_words * 4 + al((int64_t)sizeof(tg::DevParams), 16) +
                         (2 * tg::kPullMaxStages + 2) * 8 + 32 + 32;
    const int64_t room = 227 * 1024 - tail;
    int64_t ns = std::min<int64_t>(tg::kPullMaxStages, room / std::max<int64_t>(1, L.stage));
    ns -= ns % L.nteams;
    if (ns < 2 * L.nteams) return false;
    L.nstages = (int32_t)ns;
    L.idx = (int32_t)(ns * L.stage);
    L.params = (int32_t)al(L.idx + 2 * (int64_t)L.idx_words * 4, 16);
    L.mbar = (int32_t)al(L.params + (int64_t)sizeof(tg::DevParams), 16);
    L.total = L.mbar + (2 * L.nstages + 2) * 8 + 32;
    return L.total <= 227 * 1024;
}

// Builds the pull form's tables and layout for the tiles the per-step
// kernel runs; on success sets use_pull.  A scene the pull form cannot run
// is an error only when it was requested.
int setup_pull(titan_gb300_sim *s, std::vector<tg::TileInfo> &tiles_run) {
    s->use_pull = false;
    if (s->prec == P_FP64) return s->fail(TITAN_GB300_EINVAL, "the pull kernel runs FP32 and FP32C only");
    std::vector<tg::PullTile> pt(tiles_run.size());
    for (size_t t = 0; t < tiles_run.size(); t++) {
        pt[t].mass_off = tiles_run[t].mass_off;
        pt[t].ent_off = tiles_run[t].ent_off;
        pt[t].warp_off = tiles_run[t].warp_off;
        pt[t].nm = tiles_run[t].nm;
    }
    tg::PullLayout L{};
    if (!pull_layout(s->prec, tiles_run, s->threads_req, L)) {
        if (s->kernel_req == 6) return s->fail(TITAN_GB300_ELIMIT, "two tiles per team do not fit the pull kernel's shared memory");
        return TITAN_GB300_OK;
    }
    std::string why = tg::build_pull(s->plan, pt, L.team_warps, tg::state_record_bytes(s->prec) / 16,
                                     pull_springs(s), s->pull);
    if (!why.empty()) {
        s->pull = tg::PullTables();
        if (s->kernel_req == 6) return s->fail(TITAN_GB300_ELIMIT, why);
        return TITAN_GB300_OK;
    }
    s->pull_tiles = std::move(pt);
    s->args.pull = L;
    // implementation bytes of one step: state records read (tile and halo)
    // and written, m and flags per mass, the spring quads of every unit
    // (damping quads included where they are read), the tiles' actuation
    // records, unit descriptors, halo indices and tile records
    const int64_t rec = tg::state_record_bytes(s->prec);
    int64_t nh = 0, nm = 0, nact = 0, quad_bytes = 0;
    for (const tg::TileInfo &ti : tiles_run) {
        nh += ti.nh;
        nm += ti.nm;
        nact += ti.nact;
    }
    for (const tg::PullUnit &pu : s->pull.units) quad_bytes += (int64_t)pu.nquads * tg::pull_quad_bytes(pu.flags & tg::PU_DAMP);
    s->pull_impl_bytes = nm * (2 * rec + 4 + 1) + nh * (rec + 4) + quad_bytes + nact * 16 +
                         (int64_t)s->pull.units.size() * 16 + (int64_t)tiles_run.size() * (int64_t)sizeof(tg::TileInfo);
    s->use_pull = true;
    return TITAN_GB300_OK;
}

// Builds s->plan for a requested tile size (0: the default).  The default
// tile of the warp-specialised form (208 masses) gives way to 192 when two
// stages of the planned tiles would not fit one SM's shared memory.
std::string plan_scene(titan_gb300_sim *s, int tile_masses, tg::PlanInput &in) {
    s->plan_req = tile_masses;
    in = plan_input(s, tile_masses, true);
    s->plan_ask = plan_sizes(in);
    std::string why;
    if (in.tile_min < 32) {  // tiles for the resident grid, if it takes them (heavy masses may split tiles)
        int shape, stage;
        size_t bytes;
        why = tg::build_plan(in, s->plan);
        if (why.empty() && choose_grid(s, tile_infos(s->plan), shape, stage, bytes)) return why;
        in = plan_input(s, tile_masses);
    }
    why = tg::build_plan(in, s->plan);
    if (why.empty() && tile_masses == 0 && in.tile_cap == kWsDefaultTile && !pull_wanted(s)) {
        tg::WsLayout W{};
        std::vector<tg::TileInfo> tiles = tile_infos(s->plan);
        if (in.whole_cap > kWsDefaultTile)  // whole bodies above the tile size run resident
            tiles.erase(std::remove_if(tiles.begin(), tiles.end(), [](const tg::TileInfo &ti) { return ti.nh == 0; }),
                        tiles.end());
        if (!tiles.empty()) ws_stage_layout(s->prec, tiles, W);
        if (!tiles.empty() && W.nstages < 2) {
            in = plan_input(s, kWsFallbackTile);
            why = tg::build_plan(in, s->plan);
        }
    }
    return why;
}

// Doubles of one spring parameter's device array.
size_t spring_array_size(const titan_gb300_sim *s) { return (std::max<size_t>(1, (size_t)s->ns) + 31) / 32 * 32; }

// Device memory that updates of all spring parameters will still take.
size_t spring_update_bytes(const titan_gb300_sim *s) {
    if (!s->started || s->use_res || s->use_pull) return 0;
    size_t bytes = s->d_espring ? 0 : std::max<size_t>(16, s->plan.ent_spring.size() * sizeof(int32_t));
    for (int q = 0; q < titan_gb300_sim::SP_COUNT; q++) bytes += s->d_sp[q] ? 0 : spring_array_size(s) * 8;
    return bytes;
}

// Device arrays for the spring parameters of mask (a bit per SP_*), in one
// allocation (an allocation each took 10 us of a first update).
bool alloc_spring_arrays(titan_gb300_sim *s, unsigned mask, cudaError_t &e) {
    const size_t each = spring_array_size(s);
    int missing = 0;
    for (int q = 0; q < titan_gb300_sim::SP_COUNT; q++) missing += (mask >> q & 1) && !s->d_sp[q];
    if (!missing) return true;
    double *p = (double *)s->mem.get(missing * each * 8, e);
    if (!p) return false;
    for (int q = 0; q < titan_gb300_sim::SP_COUNT; q++)
        if ((mask >> q & 1) && !s->d_sp[q]) {
            s->d_sp[q] = p;
            p += each;
        }
    return true;
}

// The device's copies of the parameters of mask brought up to date with the
// host arrays.
int upload_spring_arrays(titan_gb300_sim *s, unsigned mask) {
    const std::vector<double> *host[] = {&s->k, &s->rest, &s->damping, &s->omega, &s->amp, &s->phase};
    for (int q = 0; q < titan_gb300_sim::SP_COUNT; q++) {
        if (!(mask >> q & 1)) continue;
        if (!s->sp_current[q] && !host[q]->empty())
            CK(cudaMemcpyAsync(s->d_sp[q], host[q]->data(), host[q]->size() * 8, cudaMemcpyHostToDevice, s->stream),
               "upload spring parameters");
        s->sp_current[q] = true;
    }
    return TITAN_GB300_OK;
}

// The resident grid's kernels for the current integrator made ready, so that
// step() only launches; not used where the device cannot take all its CTAs at
// once (the per-step kernels serve then, with the same tiles).
int prepare_grid(titan_gb300_sim *s) {
    if (!s->use_grid) return TITAN_GB300_OK;
    int per_sm = 0;
    CK(tg::grid_resident_prepare(s->prec, s->integrator, s->gargs, s->grid_shape, s->grid_smem, &per_sm),
       "prepare resident grid");
    if ((int64_t)s->gargs.ntiles > (int64_t)per_sm * sm_count(s)) s->use_grid = false;
    if (s->single_shape >= 0)
        CK(tg::grid_resident_prepare(s->prec, s->integrator, s->gargs, s->single_shape, s->grid_smem, &per_sm),
           "prepare resident grid");
    return TITAN_GB300_OK;
}

// The slab's records rewritten on the device for the parameters given,
// every spring's (the host loop took 1.5 ms for the 137,000 springs of a 23^3
// design).  done: false where there is no memory for it.
int refresh_entries(titan_gb300_sim *s, unsigned given, bool &done) {
    const tg::Plan &P = s->plan;
    cudaError_t e = cudaSuccess;
    done = false;
    bool room = alloc_spring_arrays(s, given, e);
    if (room && !s->d_espring) {
        std::vector<int32_t> es(P.ent_spring.begin(), P.ent_spring.end());
        room = (s->d_espring = dev_copy(s, es, e)) != nullptr;
    }
    if (!room) {
        if (e != cudaErrorMemoryAllocation) return s->cuda_fail(e, "spring parameters");
        cudaGetLastError();
        return TITAN_GB300_OK;
    }
    if (int rc = upload_spring_arrays(s, given)) return rc;
    tg::EntryArgs x{};
    x.spring = s->d_espring;
    x.rec = const_cast<void *>(s->args.ent);
    x.act = const_cast<void *>(s->args.act);
    x.count = (int64_t)P.ent_spring.size();
    for (int q = 0; q < titan_gb300_sim::SP_COUNT; q++)
        if (given >> q & 1) x.par[q] = s->d_sp[q];
    CK(tg::launch_entries(s->prec, x, s->stream), "refresh entries");
    if (s->short_form.ready)
        if (int rc = refresh_short(s)) return rc;
    s->tables_written = true;
    done = true;
    return TITAN_GB300_OK;
}

// Calls of at most this many steps run the warp-specialised kernel on tiles
// of its own size (build_short) although whole bodies are resident: a launch
// of resident bodies costs 12 to 30 us more than its steps and is bound by its
// largest bodies (a CTA of 512 masses fills an SM).  Measured, FP32C, us per
// call with resident bodies and with this: 608 bodies of 6^3 masses, 1 step 18
// and 16, 2 steps 32 and 41; of 8^3, 1 step 56 and 31, 4 steps 130 and 129;
// beside bodies too large to be resident, 320 of 6^3 to 9^3, 1 step 31 and 17,
// 6 steps 114 and 107; 600 of 3^3 to 9^3, 1 step 31 and 21, 6 steps 140 and
// 131, 12 steps 257 and 252; 1024 of 3^3 to 12^3, 1 step 94 and 71, 4 steps
// 296 and 292, 8 steps 552 and 572.
int short_limit(const titan_gb300_sim *s) {
    if (!s->use_rtiles || s->use_grid || s->prec == P_FP64 || !grid_wanted(s) || s->tile_masses > 0) return 0;
    int largest = 0;
    for (const tg::TileInfo &ti : s->rtiles) largest = std::max(largest, (int)ti.nm);
    if (largest <= kWsDefaultTile) return 0;
    if (s->args.ntiles > 0) return s->n <= 1500 * (int64_t)sm_count(s) ? 12 : 6;
    return largest <= 256 ? 1 : 4;
}

// The tables of those tiles, made at the 65th such call (or by
// prepare_steps): they take 5 to 75 ms (320 bodies of 3^3 to 9^3 11 ms, 608 of
// 8^3 61), a quarter to a half of start(), which a scene that takes a few
// short calls only would not get back.  Without room for them the resident
// bodies serve these calls too.
constexpr int64_t kShortCalls = 64;
int build_short(titan_gb300_sim *s) {
    auto &f = s->short_form;
    if (f.tried) return TITAN_GB300_OK;
    f.tried = true;
    const tg::Plan &P = s->plan;
    std::vector<tg::TileInfo> tiles;
    std::vector<int64_t> whole;
    for (const tg::TileInfo &ti : tile_infos(P)) {
        const bool cut = ti.nh == 0 && ti.nm > kWsDefaultTile;
        if (cut && ti.nheavy > 0) return TITAN_GB300_OK;
        if (cut) whole.push_back((int64_t)(std::upper_bound(P.tile_mass_off.begin(), P.tile_mass_off.end(), ti.mass_off) -
                                           P.tile_mass_off.begin()) - 1);
        else tiles.push_back(ti);
    }
    const std::vector<tg::CutTile> cuts = tg::cut_tiles(P, whole, tg::state_record_bytes(s->prec));
    // where the pieces' tables start behind the plan's
    const int64_t E = (int64_t)P.ent_ends.size();
    std::vector<int32_t> halo(P.halo), src;
    std::vector<uint32_t> warp_inc(P.warp_inc_off), ends;
    std::vector<uint16_t> inc(P.inc);
    for (const tg::CutTile &c : cuts) {
        tg::TileInfo ti{};
        ti.mass_off = (int32_t)c.lo;
        ti.nm = (int32_t)(c.hi - c.lo);
        ti.halo_off = (int32_t)halo.size();
        ti.nh = c.nh;
        ti.ent_off = (int32_t)(E + (int64_t)src.size());
        ti.ne = (int32_t)c.entry.size();
        ti.nact = c.nact;
        ti.warp_off = (int32_t)warp_inc.size();
        ti.body = c.body;
        ti.inc_off = (int32_t)inc.size();
        ti.inc_words = (int32_t)c.inc.size();
        tiles.push_back(ti);
        for (const uint32_t w : c.warp_inc) warp_inc.push_back((uint32_t)inc.size() + w);
        halo.insert(halo.end(), c.halo.begin(), c.halo.end());
        src.insert(src.end(), c.entry.begin(), c.entry.end());
        ends.insert(ends.end(), c.ends.begin(), c.ends.end());
        inc.insert(inc.end(), c.inc.begin(), c.inc.end());
    }
    if (E + src.size() > (size_t)INT32_MAX || halo.size() > (size_t)INT32_MAX || inc.size() > (size_t)INT32_MAX)
        return TITAN_GB300_OK;
    f.args = s->args;
    tg::StepArgs &a = f.args;
    ws_stage_layout(s->prec, tiles, a.ws);
    if (a.ws.nstages < 2) return TITAN_GB300_OK;
    ws_tail_layout(s->prec, a.ws);
    cudaError_t e = tg::step_ws_prepare(s->prec, tg::INTEG_EULER, (size_t)a.ws.total);
    const size_t rec = (E + src.size()) * tg::entry_record_bytes(s->prec);
    int32_t *d_src = nullptr;
    uint32_t *d_ends = nullptr;
    if (e != cudaSuccess || !(a.tiles = dev_copy(s, tiles, e)) || !(a.halo = dev_copy(s, halo, e)) ||
        !(a.warp_inc_off = dev_copy(s, warp_inc, e)) || !(a.inc = dev_copy(s, inc, e)) ||
        !(d_src = dev_copy(s, src, e)) || !(d_ends = dev_copy(s, ends, e)) || !(a.ent = s->mem.get(rec, e)) ||
        !(a.act = s->mem.get(rec, e))) {
        cudaGetLastError();
        return e == cudaErrorMemoryAllocation ? TITAN_GB300_OK : s->cuda_fail(e, "tables for calls of a few steps");
    }
    f.pieces = tg::RepeatArgs{d_src, d_ends, const_cast<void *>(a.ent), const_cast<void *>(a.act), E, (int64_t)src.size()};
    a.ntiles = (int32_t)tiles.size();
    f.ctas = (int)std::min<int64_t>((int64_t)tiles.size(), sm_count(s));
    f.ready = true;
    return refresh_short(s);
}

// The step arguments with those tables (the rest as it is now: new local
// constraints, for instance, have new arrays).
tg::StepArgs short_args(const titan_gb300_sim *s) {
    tg::StepArgs a = s->args;
    const tg::StepArgs &t = s->short_form.args;
    a.tiles = t.tiles;
    a.halo = t.halo;
    a.ent = t.ent;
    a.act = t.act;
    a.warp_inc_off = t.warp_inc_off;
    a.inc = t.inc;
    a.ntiles = t.ntiles;
    a.ws = t.ws;
    return a;
}

// Whether a call of nsteps runs in those tiles; makes their tables when there
// have been enough such calls, or at once (now).
bool short_runs(titan_gb300_sim *s, int64_t nsteps, bool now, int &rc) {
    rc = TITAN_GB300_OK;
    if (nsteps > short_limit(s)) return false;
    if (!s->short_form.tried) {
        if (!now && ++s->short_form.calls <= kShortCalls) return false;
        cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(s->stream, &st) != cudaSuccess || st != cudaStreamCaptureStatusNone) return false;
        rc = build_short(s);
    }
    return rc == TITAN_GB300_OK && s->short_form.ready;
}

// Builds the plan and all device buffers; positions/velocities come from the
// host mirror.  Keeps T / steps.
int build_device(titan_gb300_sim *s) {
    s->free_device();
    tg::PlanInput in;
    const size_t rs = s->rsize();
    // (a default plan depends on the integrator and on the form and resident
    // modes chosen: only one that these settings would ask for is taken)
    if (s->plan_adopted && !s->started && s->plan_req == s->tile_masses &&
        s->plan_ask == plan_sizes(plan_input(s, s->tile_masses, true))) {
        s->plan_adopted = false;  // the adopted plan serves this first start
        in = plan_input(s, s->plan_tile);
    } else {
        s->plan_adopted = false;
        std::string why = plan_scene(s, s->tile_masses, in);
        if (!why.empty()) return s->fail(TITAN_GB300_ELIMIT, why);
    }
    s->plan_tile = in.tile_cap;
    const tg::Plan &P = s->plan;
    // threads per CTA of the per-tile forms: one per tile mass, in FP64 two,
    // and there at least 256 while every tile gets a CTA at once (two of 256
    // threads fit one SM; tiles of 32 masses: 11.3 us per step of the 5^3
    // lattice against 12.1 with 128, 16.1 against 18.4 of a 20^3 one; with
    // more tiles the second wave costs more: 30 against 25 us at 385)
    int sms_dev = 0;
    CK(cudaDeviceGetAttribute(&sms_dev, cudaDevAttrMultiProcessorCount, s->device), "device");
    const int min_threads = s->prec == P_FP64 && P.ntiles <= 2 * sms_dev ? 256 : 128;
    s->threads = s->threads_req > 0 ? s->threads_req
                                    : std::max(min_threads, std::min(512, ((P.max_nm + 31) / 32) * 32 *
                                                                              (s->prec == P_FP64 ? 2 : 1)));
    // 96-mass FP64 tiles, three CTAs per SM: 196 us per 60^3 step with 256
    // threads, 214 with 192
    if (s->prec == P_FP64 && s->threads_req == 0 && P.max_nm > 64) s->threads = std::max(s->threads, 256);
    s->npad = ((s->n + 127) / 128) * 128;
    const int64_t np = s->npad;
    auto &a = s->args;
    a = tg::StepArgs{};
    a.npad = np;
    a.slots = std::max(P.max_slots, 1);
    a.ecap = std::max(P.max_entries, 1);
    a.hcap = std::max(P.max_heavy, 1);
    cudaError_t e = cudaSuccess;
    s->smem = 0;
    std::vector<tg::TileInfo> tiles = tile_infos(P);
    for (int64_t t = 0; t < P.ntiles; t++) {
        const tg::TileInfo &ti = tiles[t];
        // ne + 1 force slots: the last holds the zero force padding codes name
        s->smem = std::max(s->smem, s->kernel_req == 3
                                        ? tg::tile_async_smem_bytes(s->prec, ti.nm + ti.nh, ti.ne + 1, ti.nheavy)
                                        : tg::tile_smem_bytes(s->prec, ti.nm + ti.nh, ti.ne + 1, ti.nheavy));
    }
    if (P.inc.size() > (size_t)INT32_MAX) return s->fail(TITAN_GB300_ELIMIT, "incidence table exceeds 2^31 words");
    // body-resident bins: whole bodies that fit one CTA run all the steps of
    // a launch in shared memory; the per-step kernels take the other tiles
    s->use_res = false;
    s->rplan = tg::ResPlan();
    s->rargs = tg::ResArgs{};
    {
        const int cap = s->integrator == tg::INTEG_EULER ? resident_cap(s) : 0;
        if (cap > 0) {
            tg::build_resident(in, P, cap, cap, s->rplan);
            if (s->rplan.nbins > 0) {
                s->use_res = true;
                s->res_threads = s->res_threads_req > 0
                                     ? s->res_threads_req
                                     : std::max(128, std::min(512, ((cap + 1) / 2 + 31) & ~31));
                const int mpt = (cap + s->res_threads - 1) / s->res_threads;
                const size_t rsm = tg::resident_smem_bytes(s->prec, cap);
                CK(tg::resident_prepare(s->prec, mpt, rsm), "set resident shared memory");
                const int per_sm = tg::resident_ctas_per_sm(s->prec, mpt, s->res_threads, rsm);
                if (per_sm <= 0) return s->fail(TITAN_GB300_ELIMIT, "resident bins do not fit one SM");
                int sms = 0, dev = 0;
                CK(cudaGetDevice(&dev), "device");
                CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "device");
                s->res_ctas = (int)std::min<int64_t>(s->rplan.nbins, (int64_t)sms * per_sm);
                s->rargs.nbins = s->rplan.nbins;
                s->rargs.cap = cap;
            }
        }
    }
    // resident tiles: halo-free tiles run all the steps of a launch in shared
    // memory, their slab, actuation and incidence records staged there too
    // when the largest tile's fit and every tile still gets a CTA at once
    s->use_rtiles = false;
    s->rtiles.clear();
    s->rt_groups.clear();
    std::vector<uint8_t> rt_flag(P.ntiles, 0);
    // automatic: resident tiles for every halo-free tile that fits when the
    // kernel form is automatic (measured on GB300: 2.5x faster than the
    // per-step kernels on one 125-mass body, 2x on thousands of them, 5 %
    // on the 4096-body batch whose small bodies alone are halo-free;
    // never slower on the mixed scenes tried)
    const bool rt_auto = s->res_mode == -1 && s->kernel_req == 0;
    if ((s->res_mode == 2 || rt_auto) && s->integrator == tg::INTEG_EULER) {
        const size_t kMaxSmem = 227 * 1024;
        const int tcap = s->res_threads_req > 0 ? s->res_threads_req : 512;
        for (int64_t t = 0; t < P.ntiles; t++) {
            const tg::TileInfo &ti = tiles[t];
            if (ti.nh != 0 || ti.nm > tg::kResMaxMpt * tcap || tg::tile_resident_smem_bytes(s->prec, ti, 0) > kMaxSmem)
                continue;
            rt_flag[t] = 1;
            s->rtiles.push_back(ti);
        }
        // as many as the SMs or more: the largest first, in groups by size
        // with a launch each, so that small tiles get small CTAs
        auto group_of = [&](const tg::TileInfo &ti) { return ti.nm > 256 ? 0 : (ti.nm > 128 ? 1 : 2); };
        const bool many = (int64_t)s->rtiles.size() >= sms_dev && s->res_threads_req == 0;
        if (many)
            std::stable_sort(s->rtiles.begin(), s->rtiles.end(),
                             [](const tg::TileInfo &x, const tg::TileInfo &y) { return x.nm > y.nm; });
        for (size_t first = 0; first < s->rtiles.size();) {
            size_t last = first + 1;
            while (last < s->rtiles.size() && (!many || group_of(s->rtiles[last]) == group_of(s->rtiles[first]))) last++;
            titan_gb300_sim::RtGroup g;
            g.first = first;
            int64_t max_nm = 0, max_ne = 0;
            size_t sm_st = 0, sm_pl = 0;
            for (size_t q = first; q < last; q++) {
                const tg::TileInfo &ti = s->rtiles[q];
                max_nm = std::max<int64_t>(max_nm, ti.nm);
                max_ne = std::max<int64_t>(max_ne, ti.ne);
                sm_st = std::max(sm_st, tg::tile_resident_smem_bytes(s->prec, ti, 1));
                sm_pl = std::max(sm_pl, tg::tile_resident_smem_bytes(s->prec, ti, 0));
            }
            // threads: a thread per mass of the largest tile; with fewer tiles
            // than SMs, up to a quarter of its slab entries (phase B) -- in
            // [64, 512] (measured on GB300: one 125-mass tile steps fastest
            // with 288 threads, thousands of them with 128)
            const int64_t want_t = many ? max_nm : std::max<int64_t>(max_nm, max_ne / 4);
            g.threads = s->res_threads_req > 0
                            ? s->res_threads_req
                            : (int)std::max<int64_t>(64, std::min<int64_t>(512, (want_t + 31) & ~int64_t(31)));
            g.mpt = (int)((max_nm + g.threads - 1) / g.threads);
            int stage = 0;
            if (sm_st <= kMaxSmem && tg::tile_resident_prepare(s->prec, g.mpt, 1, sm_st) == cudaSuccess) {
                const int ps = tg::tile_resident_ctas_per_sm(s->prec, g.mpt, 1, g.threads, sm_st);
                stage = ps > 0 && (int64_t)(last - first) <= (int64_t)sms_dev * ps;
            }
            g.smem = stage ? sm_st : sm_pl;
            CK(tg::tile_resident_prepare(s->prec, g.mpt, stage, g.smem), "set resident-tile shared memory");
            if (tg::tile_resident_ctas_per_sm(s->prec, g.mpt, stage, g.threads, g.smem) <= 0)
                return s->fail(TITAN_GB300_ELIMIT, "resident tiles do not fit one SM");
            g.args.ntiles = (int32_t)(last - first);
            g.args.stage = stage;
            s->use_rtiles = true;
            s->rt_groups.push_back(g);
            first = last;
        }
    }
    std::vector<tg::TileInfo> tiles_run;
    for (int64_t t = 0; t < P.ntiles; t++)
        if ((!s->use_res || !s->rplan.tile_resident[t]) && !rt_flag[t]) tiles_run.push_back(tiles[t]);
    // automatic choice: the warp-specialised form in FP32 and FP32C (measured
    // fastest on GB300, see the kernel-form sweep in profiles/) when two of
    // the scene's tiles fit one SM's shared memory, else the per-tile form;
    // the per-tile form in FP64, whose CTAs overlap each other instead (three
    // per SM: 80^3 449 us per step against 496 with one)
    // the pull form when requested (or automatic, kPullAuto), else the
    // warp-specialised one
    s->use_pull = false;
    s->pull = tg::PullTables();
    s->pull_tiles.clear();
    if ((s->kernel_req == 6 || (kPullAuto && s->kernel_req == 0 && s->prec != P_FP64)) && !tiles_run.empty()) {
        int rc = setup_pull(s, tiles_run);
        if (rc) return rc;
    }
    s->use_ws = false;
    const bool want_ws =
        !s->use_pull && (s->kernel_req == 4 || (s->kernel_req == 0 && s->prec != P_FP64 && !tiles_run.empty()));
    if (want_ws) {
        tg::WsLayout &W = a.ws;
        ws_stage_layout(s->prec, tiles_run, W);
        if (W.nstages < 2 && s->kernel_req == 4)
            return s->fail(TITAN_GB300_ELIMIT, "two tiles do not fit in shared memory for the warp-specialised kernel");
    }
    if (want_ws && a.ws.nstages >= 2) {
        tg::WsLayout &W = a.ws;
        ws_tail_layout(s->prec, W);
        s->ws_warps = s->threads_req > 0 ? s->threads_req / 32 : tg::kWsMaxConsumerWarps;
        s->ws_warps = std::max(2, std::min(tg::kWsMaxConsumerWarps, s->ws_warps)) & ~1;
        CK(tg::step_ws_prepare(s->prec, s->integrator, (size_t)W.total), "set shared memory");
        int sms = 0, dev = 0;
        CK(cudaGetDevice(&dev), "device");
        CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "device");
        s->ctas = (int)std::min<int64_t>((int64_t)tiles_run.size(), sms);
        s->threads = (s->ws_warps + tg::kWsProducerWarps) * 32;
        s->use_ws = true;
    }
    if (s->use_pull) {
        CK(tg::step_pull_prepare(s->prec, s->integrator, (size_t)a.pull.total), "set shared memory");
        int sms = 0, dev = 0;
        CK(cudaGetDevice(&dev), "device");
        CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "device");
        s->ctas = (int)std::min<int64_t>((int64_t)tiles_run.size(), sms);
        s->threads = (a.pull.nteams * a.pull.team_warps + 1) * 32;
    } else if (!s->use_ws) {
        if (s->smem > 227 * 1024) return s->fail(TITAN_GB300_ELIMIT, "tile does not fit in shared memory");
        s->use_async = s->kernel_req == 3;
        s->step_variant = 0;
        if (s->min_ctas_req >= 3 && s->prec != P_FP64) {
            if (s->threads > 256)
                return s->fail(TITAN_GB300_EINVAL, "3 or 4 CTAs per SM need at most 256 threads per CTA");
            s->step_variant = s->min_ctas_req == 3 ? 1 : 2;
        }
        // capped registers, which spill, only where three CTAs' shared memory
        // fits an SM: 60^3 with tiles of 128 masses 222 us with the cap and 215
        // without, of 192 302 and 278
        const bool three = 3 * (s->smem + 1024) <= 228 * 1024;
        if (s->prec == P_FP64 && s->threads <= 256 && three && (int64_t)tiles_run.size() > 2 * sms_dev)
            s->step_variant = 3;
        if (s->use_async)
            CK(tg::step_async_prepare(s->prec, s->smem), "set shared memory");
        else
            CK(tg::step_prepare(s->prec, s->step_variant, s->integrator, s->smem), "set shared memory");
    }
    a.ntiles = (int32_t)tiles_run.size();
    if (P.ent_ends.size() > (size_t)INT32_MAX || P.halo.size() > (size_t)INT32_MAX)
        return s->fail(TITAN_GB300_ELIMIT, "more than 2^31 slab entries");
#define DEVCOPY(dst, vec, what)                               \
    do {                                                      \
        auto *p_ = dev_copy(s, vec, e);                       \
        if (!p_) return s->cuda_fail(e, what);                \
        dst = p_;                                             \
    } while (0)
    DEVCOPY(a.tiles, tiles_run, "upload tiles");
    if (s->use_pull) {
        DEVCOPY(a.pull_units, s->pull.units, "upload pull units");
        DEVCOPY(a.pull_ell, s->pull.ell, "upload pull columns");
    }
    if (s->use_rtiles) {
        tg::TileInfo *rt = nullptr;
        DEVCOPY(rt, s->rtiles, "upload resident tiles");
        for (auto &g : s->rt_groups) g.args.tiles = rt + g.first;
    }
    if (s->use_res) {
        tg::ResPlan &R = s->rplan;
        tg::ResArgs &r = s->rargs;
        DEVCOPY(r.bin_mass_off, R.bin_mass_off, "upload bins");
        DEVCOPY(r.bin_warp_off, R.bin_warp_off, "upload bins");
        DEVCOPY(r.mass, R.mass, "upload bins");
        DEVCOPY(r.body, R.body, "upload bins");
        DEVCOPY(r.deg, R.deg, "upload bins");
        DEVCOPY(r.act_mask, R.act_mask, "upload bins");
        DEVCOPY(r.warp_rec_off, R.warp_rec_off, "upload bins");
        const size_t nrec = std::max<size_t>(1, R.words.size()) * (s->prec == P_FP64 ? 32 : 16);
        if (!(r.rec = s->mem.get(nrec, e))) return s->cuda_fail(e, "alloc resident records");
        if (!(r.act = s->mem.get(nrec, e))) return s->cuda_fail(e, "alloc resident records");
        if (!(r.next = (int *)s->mem.get(sizeof(int), e))) return s->cuda_fail(e, "alloc bin queue");
    }
    DEVCOPY(a.halo, P.halo, "upload halo");
    s->gargs = tg::GridResArgs{};
    s->gargs.last_poll = (s->wait_polls > 0 ? (uint32_t)s->wait_polls : tg::kGridPolls) - 1;
    s->single_shape = -1;
    s->grid_last = 0;
    s->use_grid = !tiles_run.empty() && grid_wanted(s) && !s->use_pull &&
                  choose_grid(s, tiles, s->grid_shape, s->gargs.stage, s->grid_smem);
    if (s->use_grid) {
        s->gargs.ntiles = (int32_t)tiles.size();
        s->gargs.max_nm = P.max_nm;
        std::vector<int32_t> halo(P.halo);
        std::vector<uint8_t> exported(np, 0);
        for (int32_t &h : halo) {
            if (!s->fixed.empty() && s->fixed[P.new2old[h]]) h = -1;
            else exported[h] = 1;
        }
        if (s->prec != P_FP64 && s->gargs.stage && P.max_nm <= kSingleMasses &&
            (int64_t)tiles.size() <= (int64_t)sms_dev * tg::grid_resident_ctas(kSingleShape))
            s->single_shape = kSingleShape;
        if (s->use_rtiles) DEVCOPY(s->gargs.tiles, tiles, "upload tiles");
        else s->gargs.tiles = a.tiles;
        DEVCOPY(s->gargs.halo, halo, "upload halo");
        DEVCOPY(s->gargs.exported, exported, "upload exported masses");
        s->gargs.xbytes = np * tg::grid_resident_exchange_bytes(s->prec);
        if (!(s->gargs.xbuf = (uint8_t *)s->mem.get(2 * s->gargs.xbytes, e))) return s->cuda_fail(e, "alloc exchange");
        CK(cudaMemset(s->gargs.xbuf, 0, 2 * s->gargs.xbytes), "clear exchange");
        if (int rc = prepare_grid(s)) return rc;
    }
    DEVCOPY(a.warp_inc_off, P.warp_inc_off, "upload warp offsets");
    std::vector<uint8_t> deg(np, 0);
    std::copy(P.deg.begin(), P.deg.end(), deg.begin());
    DEVCOPY(a.deg, deg, "upload degrees");
    DEVCOPY(a.inc, P.inc, "upload incidence");
    DEVCOPY(a.heavy_local, P.heavy_local, "upload heavy");
    DEVCOPY(a.heavy_inc_off, P.heavy_inc_off, "upload heavy");
    DEVCOPY(a.heavy_inc, P.heavy_inc, "upload heavy");
    DEVCOPY(s->d_old2new, P.old2new, "upload order");
    std::vector<double> bp(6 * std::max<size_t>(1, s->body_plane.size()), 0.0);
    for (size_t b = 0; b < s->body_plane.size(); b++)
        for (int c = 0; c < 6; c++) bp[6 * b + c] = s->body_plane[b][c];
    std::vector<float> bpf(bp.begin(), bp.end());
    DEVCOPY(a.body_plane, bp, "upload body planes");
    DEVCOPY(a.body_planef, bpf, "upload body planes");
#undef DEVCOPY
    const size_t E = std::max<size_t>(1, P.ent_ends.size());
    const size_t rs4 = (s->prec == P_FP64 ? 32 : 16);
    if (!(a.ent = s->mem.get(E * rs4, e))) return s->cuda_fail(e, "alloc entries");
    if (!(a.act = s->mem.get(E * rs4, e))) return s->cuda_fail(e, "alloc actuation");
    if (!(a.mass = s->mem.get(np * rs, e))) return s->cuda_fail(e, "alloc mass");
    if (!(a.flags = (const uint8_t *)s->mem.get(np, e))) return s->cuda_fail(e, "alloc flags");
    if (!(a.ext = s->mem.get(3 * np * rs, e))) return s->cuda_fail(e, "alloc ext");
    if (!(a.drag = (const int32_t *)s->mem.get(np * 4, e))) return s->cuda_fail(e, "alloc drag");
    if (!(a.lc_ptr = (const int32_t *)s->mem.get((np + 1) * 4, e))) return s->cuda_fail(e, "alloc lc");
    if (!(a.state0 = s->mem.get(s->comps() * np * rs, e))) return s->cuda_fail(e, "alloc state");
    if (!(a.state1 = s->mem.get(s->comps() * np * rs, e))) return s->cuda_fail(e, "alloc state");
    if (!(a.acc = s->mem.get(3 * np * rs, e))) return s->cuda_fail(e, "alloc acc");
    if (!(a.tbuf = (double *)s->mem.get(2 * sizeof(double), e))) return s->cuda_fail(e, "alloc time");
    if (s->use_rtiles) {
        if (!(s->d_t0 = (double *)s->mem.get(sizeof(double), e))) return s->cuda_fail(e, "alloc time");
        if (!s->ev_fork) CK(cudaEventCreateWithFlags(&s->ev_fork, cudaEventDisableTiming), "create event");
        for (size_t q = 0; q < s->rt_groups.size(); q++) {
            if (!s->side_stream[q])
                CK(cudaStreamCreateWithFlags(&s->side_stream[q], cudaStreamNonBlocking), "create stream");
            if (!s->ev_join[q]) CK(cudaEventCreateWithFlags(&s->ev_join[q], cudaEventDisableTiming), "create event");
        }
    }
    if (!(s->dprm = (tg::DevParams *)s->mem.get(sizeof(tg::DevParams), e))) return s->cuda_fail(e, "alloc params");
    a.prm = s->dprm;
    if (!(s->d_err = (int *)s->mem.get(sizeof(int), e))) return s->cuda_fail(e, "alloc error flag");
    CK(cudaMemset(s->d_err, 0, sizeof(int)), "clear error flag");
    a.err = s->d_err;
    if (!(s->d_xfer = (double *)s->mem.get(9 * (size_t)s->n * 8, e))) return s->cuda_fail(e, "alloc staging");
    if (!(s->d_idx = (int64_t *)s->mem.get((size_t)s->n * 8, e))) return s->cuda_fail(e, "alloc staging");
    CK(cudaMallocHost(&s->h_xfer, 9 * (size_t)s->n * 8 + 16), "alloc pinned staging");
    CK(cudaHostGetDevicePointer((void **)&s->stage_dev, s->h_xfer, 0), "map pinned staging");
    CK(tg::xfer_prepare(s->prec), "load transfer kernels");
    s->h_err = reinterpret_cast<int *>(s->h_xfer + 9 * s->n);
    CK(cudaMemset(a.state0, 0, s->comps() * np * rs), "clear state");
    CK(cudaMemset(a.state1, 0, s->comps() * np * rs), "clear state");
    CK(cudaMemset(a.acc, 0, 3 * np * rs), "clear acc");

    int rc = upload_entries(s);
    if (rc) return rc;
    rc = upload_mass_attrs(s);
    if (rc) return rc;
    // positions / velocities into both ping-pong buffers
    std::memcpy(s->h_xfer, s->pos.data(), 3 * s->n * 8);
    std::memcpy(s->h_xfer + 3 * s->n, s->vel.data(), 3 * s->n * 8);
    CK(cudaMemcpy(s->d_xfer, s->h_xfer, 6 * s->n * 8, cudaMemcpyHostToDevice), "upload state");
    tg::XferArgs x{};
    x.old2new = s->d_old2new;
    x.count = s->n;
    x.npad = np;
    x.state0 = a.state0;
    x.state1 = a.state1;
    x.acc = a.acc;
    x.ipos = s->d_xfer;
    x.ivel = s->d_xfer + 3 * s->n;
    CK(tg::launch_scatter(s->prec, x, s->stream), "scatter state");
    s->parity = 0;
    rc = upload_params(s);
    if (rc) return rc;
    CK(cudaStreamSynchronize(s->stream), "start");
    return TITAN_GB300_OK;
}

// Downloads positions/velocities into the host mirror (creation order).
int pull_state(titan_gb300_sim *s) {
    tg::XferArgs x{};
    x.old2new = s->d_old2new;
    x.count = s->n;
    x.npad = s->npad;
    x.state0 = s->args.state0;
    x.state1 = s->args.state1;
    x.acc = s->args.acc;
    x.parity = s->parity;
    x.pos = s->d_xfer;
    x.vel = s->d_xfer + 3 * s->n;
    CK(tg::launch_gather(s->prec, x, s->stream), "gather state");
    CK(cudaMemcpyAsync(s->h_xfer, s->d_xfer, 6 * s->n * 8, cudaMemcpyDeviceToHost, s->stream), "download");
    CK(cudaStreamSynchronize(s->stream), "download");
    std::memcpy(s->pos.data(), s->h_xfer, 3 * s->n * 8);
    std::memcpy(s->vel.data(), s->h_xfer + 3 * s->n, 3 * s->n * 8);
    return TITAN_GB300_OK;
}

// Per-mass local time: the reference adds dt to each free mass every step
// (src/sim.cu:1165); replay those additions from the mass's last upload.
void mass_times(titan_gb300_sim *s, const int64_t *idx, int64_t count, double *T) {
    std::map<std::pair<uint64_t, int64_t>, double> memo;
    for (int64_t q = 0; q < count; q++) {
        int64_t i = idx ? idx[q] : q;
        if (!s->fixed.empty() && s->fixed[i]) {
            T[q] = s->mT0[i];
            continue;
        }
        uint64_t bits;
        std::memcpy(&bits, &s->mT0[i], 8);
        auto key = std::make_pair(bits, s->mTstep[i]);
        auto it = memo.find(key);
        if (it != memo.end()) {
            T[q] = it->second;
            continue;
        }
        double t = s->mT0[i];
        int64_t st = s->mTstep[i];
        for (size_t r = 0; r < s->dt_log.size(); r++) {
            int64_t b = s->dt_log[r].first;
            int64_t e = r + 1 < s->dt_log.size() ? s->dt_log[r + 1].first : s->steps;
            double d = s->dt_log[r].dt;
            if (s->dt_log[r].halves == 2) {  // RK2: mass.T += 0.5 * dt twice per step
                const double h = 0.5 * d;
                for (int64_t z = std::max(b, st); z < e; z++) {
                    t = t + h;
                    t = t + h;
                }
                continue;
            }
            for (int64_t z = std::max(b, st); z < e; z++) t = t + d;
        }
        memo[key] = t;
        T[q] = t;
    }
}

cudaGraphExec_t get_graph(titan_gb300_sim *s, int len, int parity, cudaError_t &e) {
    auto key = std::make_pair(len, parity);
    auto it = s->graphs.find(key);
    if (it != s->graphs.end()) return it->second;
    cudaGraph_t g = nullptr;
    e = cudaStreamBeginCapture(s->stream, cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) return nullptr;
    int p = parity;
    cudaError_t el = cudaSuccess;  // the first launch refused while capturing
    const bool written = s->tables_written;
    s->tables_written = false;  // the graph's first step starts after all work before it
    for (int i = 0; i < len; i++)
        for (int q = 0; q < s->passes(); q++) {
            const cudaError_t r = s->launch(p, 0, q);
            if (el == cudaSuccess) el = r;
            p ^= 1;
        }
    s->tables_written = written;
    e = cudaStreamEndCapture(s->stream, &g);
    if (e == cudaSuccess && el != cudaSuccess) {
        cudaGraphDestroy(g);
        e = el;
    }
    if (e != cudaSuccess) return nullptr;
    cudaGraphExec_t ex = nullptr;
    e = cudaGraphInstantiate(&ex, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) return nullptr;
    s->graphs[key] = ex;
    return ex;
}

bool ensure_device(titan_gb300_sim *s) { return cudaSetDevice(s->device) == cudaSuccess; }

// Whether this call of step() is one resident-grid launch: two steps or more
// (a launch stages the tiles' tables once).  Under stream capture the
// per-step path decides, as without the resident grid.
bool grid_runs(titan_gb300_sim *s, int64_t nsteps) {
    if (!s->use_grid || nsteps < kGridMinSteps) return false;
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    return cudaStreamIsCapturing(s->stream, &st) == cudaSuccess && st == cudaStreamCaptureStatusNone;
}

// Whether this call is a single step that runs as one pass of the resident
// grid's kernel.
bool single_runs(titan_gb300_sim *s, int64_t nsteps) {
    if (!s->use_grid || s->single_shape < 0 || nsteps != 1) return false;
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    return cudaStreamIsCapturing(s->stream, &st) == cudaSuccess && st == cudaStreamCaptureStatusNone;
}

// The host's clock and step count after nsteps steps.
void advance_clock(titan_gb300_sim *s, int64_t nsteps) {
    if (s->passes() == 2) {
        const double h = 0.5 * s->dt;
        for (int64_t i = 0; i < nsteps; i++) {  // src/sim.cu:1574-1583
            s->T = s->T + h;
            s->T = s->T + h;
        }
    } else {
        for (int64_t i = 0; i < nsteps; i++) s->T = s->T + s->dt;  // src/sim.cu:1590
    }
    s->steps += nsteps;
}

// After a synchronisation: did a step kernel give up a bounded wait?
int check_kernel_error(titan_gb300_sim *s) {
    if (!s->d_err) return TITAN_GB300_OK;
    int flag = 0;
    CK(cudaMemcpy(&flag, s->d_err, sizeof(int), cudaMemcpyDeviceToHost), "read error flag");
    if (flag) {
        cudaMemset(s->d_err, 0, sizeof(int));
        s->torn = true;
        return s->fail(TITAN_GB300_ETIMEOUT,
                       "a step kernel's bounded wait (for its shared-memory copies or for other tiles' masses) timed out");
    }
    return TITAN_GB300_OK;
}

}  // namespace

namespace tg {

int serve_begin(titan_gb300_sim *s, int device, int precision, size_t tile_smem, ServeScene &v, std::string &why) {
    if (!s->started) return why = "the scene has not started", TITAN_GB300_ESTATE;
    if (s->serving) return why = "the scene is already with a server", TITAN_GB300_ESTATE;
    if (s->device != device || s->prec != precision)
        return why = "the scene's device or precision differs from the server's", TITAN_GB300_EINVAL;
    if (s->integrator != INTEG_EULER) return why = "the server steps symplectic Euler only", TITAN_GB300_EINVAL;
    if (s->torn) return why = "the scene's state is undefined since a step kernel's wait timed out", TITAN_GB300_ETIMEOUT;
    if (s->use_res || s->use_rtiles || s->args.ntiles <= 0)
        return why = "start the scene with resident tiles and bins off (set_resident 0)", TITAN_GB300_EINVAL;
    size_t need = 0;
    for (const TileInfo &ti : tile_infos(s->plan))
        need = std::max(need, tile_smem_bytes(s->prec, ti.nm + ti.nh, ti.ne + 1, ti.nheavy));
    if (need > tile_smem)
        return why = "a tile needs more shared memory than the server has (plan smaller tiles)", TITAN_GB300_ELIMIT;
    if (!ensure_device(s)) return why = "cudaSetDevice failed", TITAN_GB300_ECUDA;
    const cudaError_t e = cudaStreamSynchronize(s->stream);
    if (e != cudaSuccess) return why = std::string("scene stream: ") + cudaGetErrorString(e), TITAN_GB300_ECUDA;
    s->serving = true;
    v.args = &s->args;
    v.parity = s->parity;
    return TITAN_GB300_OK;
}

void serve_end(titan_gb300_sim *s, int64_t nsteps) {
    s->serving = false;
    if (nsteps <= 0) return;
    s->parity ^= (int)(nsteps & 1);
    for (int64_t i = 0; i < nsteps; i++) s->T = s->T + s->dt;  // src/sim.cu:1590
    s->steps += nsteps;
}

}  // namespace tg

// Status of a C++ exception that reached an entry point (a host allocation
// that failed, or a library error): the C ABI throws nothing, and the
// message goes to the handle when there is one.
static int host_exception(titan_gb300_sim *s) noexcept {
    int code = TITAN_GB300_EINVAL;
    std::string msg = "host error";
    try {
        throw;
    } catch (const std::bad_alloc &) {
        code = TITAN_GB300_ENOMEM;
        msg = "host memory exhausted";
    } catch (const std::exception &e) {
        try {
            msg = std::string("host error: ") + e.what();
        } catch (...) {
        }
    } catch (...) {
    }
    if (s) {
        try {
            s->err = msg;
        } catch (...) {
        }
    }
    return code;
}

extern "C" {

const char *titan_gb300_version(void) { return "titan_gb300 0.1 (sm_103a)"; }

int titan_gb300_create(titan_gb300_sim **out, int device, int precision) try {
    if (!out) return TITAN_GB300_EINVAL;
    *out = nullptr;
    if (precision < 0 || precision > 2 || device < 0) return TITAN_GB300_EINVAL;
    // No CUDA call here: the device and stream are taken at start(), so a
    // scene can be built and planned on a host without a GPU.
    auto *s = new (std::nothrow) titan_gb300_sim();
    if (!s) return TITAN_GB300_ENOMEM;
    s->device = device;
    s->prec = precision;
    *out = s;
    return TITAN_GB300_OK;
} catch (...) {
    return host_exception(nullptr);
}

void titan_gb300_destroy(titan_gb300_sim *s) {
    if (!s) return;
    if (s->stream) ensure_device(s);
    delete s;
}

int titan_gb300_set_launch(titan_gb300_sim *s, int threads_per_cta) try {
    if (!s) return TITAN_GB300_EINVAL;
    if (threads_per_cta != 0 && (threads_per_cta < 64 || threads_per_cta > 512 || threads_per_cta % 32))
        return s->fail(TITAN_GB300_EINVAL, "threads per CTA must be 0 or a multiple of 32 in [64, 512]");
    if (s->started) return s->fail(TITAN_GB300_ESTATE, "set the launch shape before start");
    s->threads_req = threads_per_cta;
    return TITAN_GB300_OK;
} catch (...) {
    return host_exception(s);
}

int titan_gb300_set_occupancy(titan_gb300_sim *s, int min_ctas_per_sm) try {
    if (!s) return TITAN_GB300_EINVAL;
    if (min_ctas_per_sm < 0 || min_ctas_per_sm > 4 || min_ctas_per_sm == 2)
        return s->fail(TITAN_GB300_EINVAL, "minimum CTAs per SM must be 0, 1, 3 or 4");
    if (s->started) return s->fail(TITAN_GB300_ESTATE, "set the occupancy before start");
    s->min_ctas_req = min_ctas_per_sm;
    return TITAN_GB300_OK;
} catch (...) {
    return host_exception(s);
}

int titan_gb300_set_kernel(titan_gb300_sim *s, int variant) try {
    if (!s) return TITAN_GB300_EINVAL;
    if (variant < 0 || variant > 6 || variant == 2 || variant == 5)
        return s->fail(TITAN_GB300_EINVAL, "kernel variant must be 0, 1, 3, 4 or 6");
    if (s->started) return s->fail(TITAN_GB300_ESTATE, "choose the kernel before start");
    s->kernel_req = variant;
    return TITAN_GB300_OK;
} catch (...) {
    return host_exception(s);
}

int titan_gb300_kernel_info(const titan_gb300_sim *s, int64_t out[4]) {
    if (!s || !out) return TITAN_GB300_EINVAL;
    if (s->use_rtiles && s->args.ntiles == 0) {
        out[0] = 5;
        out[1] = (int64_t)s->rtiles.size();
        out[2] = s->rt_groups[0].threads;
        out[3] = (int64_t)s->rt_groups[0].smem;
        return TITAN_GB300_OK;
    }
    out[0] = s->use_pull ? 6 : (s->use_async ? 3 : (s->use_ws ? 4 : 1));
    out[1] = (s->use_ws || s->use_pull) ? s->ctas : s->args.ntiles;
    out[2] = s->threads;
    out[3] = s->use_pull ? s->args.pull.total : (s->use_ws ? s->args.ws.total : (int64_t)s->smem);
    return TITAN_GB300_OK;
}

int titan_gb300_set_resident(titan_gb300_sim *s, int mode, int bin_masses, int threads_per_cta) try {
    if (!s) return TITAN_GB300_EINVAL;
    if (mode < -1 || mode > 2) return s->fail(TITAN_GB300_EINVAL, "resident mode must be -1, 0, 1 or 2");
    if (bin_masses < 0 || bin_masses > 32767) return s->fail(TITAN_GB300_EINVAL, "bin size must be in [0, 32767]");
    if (threads_per_cta != 0 && (threads_per_cta < 64 || threads_per_cta > 512 || threads_per_cta % 32))
        return s->fail(TITAN_GB300_EINVAL, "threads per CTA must be 0 or a multiple of 32 in [64, 512]");
    if (s->started) return s->fail(TITAN_GB300_ESTATE, "configure resident bins before start");
    s->res_mode = mode;
    s->res_bin_req = bin_masses;
    s->res_threads_req = threads_per_cta;
    return TITAN_GB300_OK;
} catch (...) {
    return host_exception(s);
}

int titan_gb300_resident_info(const titan_gb300_sim *s, int64_t out[8]) {
    if (!s || !out) return TITAN_GB300_EINVAL;
    std::memset(out, 0, 8 * sizeof(int64_t));
    if (s->use_rtiles) {
        out[0] = 2;
        out[1] = (int64_t)s->rtiles.size();
        std::vector<int32_t> bodies;
        int64_t nm = 0, cap = 0;
        for (const tg::TileInfo &ti : s->rtiles) {
            bodies.push_back(ti.body);
            nm += ti.nm;
            cap = std::max<int64_t>(cap, ti.nm);
        }
        std::sort(bodies.begin(), bodies.end());
        out[2] = (int64_t)(std::unique(bodies.begin(), bodies.end()) - bodies.begin());
        out[3] = nm;
        out[4] = cap;
        out[5] = s->rt_groups[0].threads;
        out[6] = (int64_t)s->rtiles.size();
        out[7] = (int64_t)s->rt_groups[0].smem;
        return TITAN_GB300_OK;
    }
    if (!s->use_res) return TITAN_GB300_OK;
    out[0] = 1;
    out[1] = s->rplan.nbins;
    out[2] = s->rplan.nbodies;
    out[3] = s->rplan.nmasses;
    out[4] = s->rargs.cap;
    out[5] = s->res_threads;
    out[6] = s->res_ctas;
    out[7] = (int64_t)tg::resident_smem_bytes(s->prec, s->rargs.cap);
    return TITAN_GB300_OK;
}

int titan_gb300_set_wait_limit(titan_gb300_sim *s, int64_t polls) {
    if (!s) return TITAN_GB300_EINVAL;
    if (polls < 0 || polls > (int64_t)UINT32_MAX) return s->fail(TITAN_GB300_EINVAL, "polls must be in [0, 2^32)");
    s->wait_polls = polls;
    s->gargs.last_poll = (polls > 0 ? (uint32_t)polls : tg::kGridPolls) - 1;
    return TITAN_GB300_OK;
}

int titan_gb300_grid_info(const titan_gb300_sim *s, int64_t out[8]) {
    if (!s || !out) return TITAN_GB300_EINVAL;
    std::fill(out, out + 8, 0);
    if (!s->started) return TITAN_GB300_OK;
    out[7] = s->grid_last;
    if (!s->use_grid) return TITAN_GB300_OK;
    out[0] = 1;
    out[1] = s->gargs.ntiles;
    out[2] = tg::grid_resident_threads(s->grid_shape);
    out[3] = (int64_t)s->grid_smem;
    out[4] = s->gargs.stage;
    out[5] = tg::grid_resident_lanes(s->prec, s->grid_shape, s->gargs.max_nm);
    out[6] = s->single_shape >= 0;
    return TITAN_GB300_OK;
}

int titan_gb300_adopt_plan(titan_gb300_sim *s, const titan_gb300_sim *src) try {
    if (!s || !src) return TITAN_GB300_EINVAL;
    if (s->started) return s->fail(TITAN_GB300_ESTATE, "adopt a plan before start");
    if (src->plan.ntiles <= 0) return s->fail(TITAN_GB300_EINVAL, "the source handle has no plan");
    auto flags = [](const titan_gb300_sim *h, int64_t i) { return !h->fixed.empty() && h->fixed[i] != 0; };
    auto act = [](const titan_gb300_sim *h, int64_t j) { return !h->type.empty() && h->type[j] >= 2; };
    bool same = s->prec == src->prec && s->n == src->n && s->ns == src->ns && s->left == src->left &&
                s->right == src->right && s->body_ptr == src->body_ptr && s->kernel_req == src->kernel_req;
    for (int64_t i = 0; same && i < s->n; i++) same = flags(s, i) == flags(src, i);
    for (int64_t j = 0; same && j < s->ns; j++) same = act(s, j) == act(src, j);
    if (!same)
        return s->fail(TITAN_GB300_EINVAL,
                       "adopt_plan needs the same precision, kernel form, masses, springs, fixed masses, "
                       "actuated springs and bodies");
    s->plan = src->plan;
    s->plan_tile = src->plan_tile;
    s->plan_req = src->plan_req;
    s->plan_ask = src->plan_ask;
    s->plan_adopted = true;
    return TITAN_GB300_OK;
} catch (...) {
    return host_exception(s);
}

int titan_gb300_plan_host(titan_gb300_sim *s, int tile_masses) try {
    if (!s) return TITAN_GB300_EINVAL;
    if (s->started) return s->fail(TITAN_GB300_ESTATE, "plan_host is for scenes that have not started");
    if (s->n <= 0) return s->fail(TITAN_GB300_EINVAL, "no masses");
    tg::PlanInput in;
    std::string why = plan_scene(s, tile_masses, in);
    if (!why.empty()) return s->fail(TITAN_GB300_ELIMIT, why);
    s->plan_tile = in.tile_cap;
    s->plan_adopted = false;
    s->rplan = tg::ResPlan();
    const int cap = resident_cap(s);
    if (cap > 0) tg::build_resident(in, s->plan, cap, cap, s->rplan);
    return TITAN_GB300_OK;
} catch (...) {
    return host_exception(s);
}

int64_t titan_gb300_plan_table(const titan_gb300_sim *s, int table, void *out) {
    if (!s) return -1;
    const tg::Plan &P = s->plan;
    auto put = [&](const auto &v) -> int64_t {
        if (out && !v.empty()) std::memcpy(out, v.data(), v.size() * sizeof(v[0]));
        return (int64_t)v.size();
    };
    switch (table) {
        case TITAN_GB300_T_NEW2OLD: return put(P.new2old);
        case TITAN_GB300_T_TILE_MASS_OFF: return put(P.tile_mass_off);
        case TITAN_GB300_T_TILE_HALO_OFF: return put(P.tile_halo_off);
        case TITAN_GB300_T_HALO: return put(P.halo);
        case TITAN_GB300_T_TILE_ENT_OFF: return put(P.tile_ent_off);
        case TITAN_GB300_T_TILE_NACT: return put(P.tile_nact);
        case TITAN_GB300_T_ENT_ENDS: return put(P.ent_ends);
        case TITAN_GB300_T_ENT_SPRING: return put(P.ent_spring);
        case TITAN_GB300_T_TILE_WARP_OFF: return put(P.tile_warp_off);
        case TITAN_GB300_T_WARP_INC_OFF: return put(P.warp_inc_off);
        case TITAN_GB300_T_DEG: return put(P.deg);
        case TITAN_GB300_T_INC: return put(P.inc);
        case TITAN_GB300_T_TILE_HEAVY_OFF: return put(P.tile_heavy_off);
        case TITAN_GB300_T_HEAVY_LOCAL: return put(P.heavy_local);
        case TITAN_GB300_T_HEAVY_INC_OFF: return put(P.heavy_inc_off);
        case TITAN_GB300_T_HEAVY_INC: return put(P.heavy_inc);
        case TITAN_GB300_T_BODY_OF_TILE: return put(P.body_of_tile);
        case TITAN_GB300_T_TILE_NH: return put(P.tile_nh);
        case TITAN_GB300_T_RES_BIN_MASS_OFF: return put(s->rplan.bin_mass_off);
        case TITAN_GB300_T_RES_BIN_WARP_OFF: return put(s->rplan.bin_warp_off);
        case TITAN_GB300_T_RES_MASS: return put(s->rplan.mass);
        case TITAN_GB300_T_RES_BODY: return put(s->rplan.body);
        case TITAN_GB300_T_RES_DEG: return put(s->rplan.deg);
        case TITAN_GB300_T_RES_ACT_MASK: return put(s->rplan.act_mask);
        case TITAN_GB300_T_RES_WARP_REC_OFF: return put(s->rplan.warp_rec_off);
        case TITAN_GB300_T_RES_WORDS: return put(s->rplan.words);
        case TITAN_GB300_T_RES_REC_SPRING: return put(s->rplan.rec_spring);
        case TITAN_GB300_T_RES_RESIDENT: return put(s->rplan.resident);
        default: return -1;
    }
}

const char *titan_gb300_last_error(const titan_gb300_sim *s) {
    return s ? s->err.c_str() : "null handle";
}

int titan_gb300_set_masses(titan_gb300_sim *s, int64_t n, const double *pos, const double *vel,
                           const double *m, const double *ext, const uint8_t *fixed, const double *drag) try {
    if (!s) return TITAN_GB300_EINVAL;
    s->plan_adopted = false;  // the topology may change
    if (s->started) return s->fail(TITAN_GB300_ESTATE, "masses can only be replaced before start");
    if (n <= 0 || !pos || !m) return s->fail(TITAN_GB300_EINVAL, "need n > 0, pos and m");
    s->n = n;
    s->pos.assign(pos, pos + 3 * n);
    s->vel.assign(3 * n, 0.0);
    if (vel) s->vel.assign(vel, vel + 3 * n);
    s->m.assign(m, m + n);
    s->ext.clear();
    if (ext) s->ext.assign(ext, ext + 3 * n);
    s->fixed.clear();
    if (fixed) s->fixed.assign(fixed, fixed + n);
    s->drag.clear();
    if (drag) {
        s->drag.resize(n);
        for (int64_t i = 0; i < n; i++) s->drag[i] = (int32_t)drag[i];  // object.h:213 truncation
    }
    s->lc_ptr.clear();
    s->lc_type.clear();
    s->lc_rec.clear();
    return TITAN_GB300_OK;
} catch (...) {
    return host_exception(s);
}

int titan_gb300_set_springs(titan_gb300_sim *s, int64_t n, const int32_t *left, const int32_t *right,
                            const double *k, const double *rest, const double *damping,
                            const int32_t *type, const double *omega, const double *amp,
                            const double *phase) try {
    if (!s) return TITAN_GB300_EINVAL;
    s->plan_adopted = false;  // the topology may change
    if (s->started) return s->fail(TITAN_GB300_ESTATE, "springs can only be replaced before start");
    if (n < 0 || (n > 0 && (!left || !right || !k || !rest))) return s->fail(TITAN_GB300_EINVAL, "bad springs");
    s->ns = n;
    s->left.assign(left, left + n);
    s->right.assign(right, right + n);
    s->k.assign(k, k + n);
    s->rest.assign(rest, rest + n);
    s->damping.assign(n, 0.0);
    if (damping) s->damping.assign(damping, damping + n);
    s->type.clear();
    if (type) {
        s->type.assign(type, type + n);
        for (int32_t t : s->type)
            if (t < 0 || t > 3) return s->fail(TITAN_GB300_EINVAL, "spring type must be 0..3");
    }
    s->omega.clear();
    if (omega) s->omega.assign(omega, omega + n);
    s->amp.clear();
    if (amp) s->amp.assign(amp, amp + n);
    s->phase.clear();
    if (phase) s->phase.assign(phase, phase + n);
    return TITAN_GB300_OK;
} catch (...) {
    return host_exception(s);
}

int titan_gb300_set_local_constraints(titan_gb300_sim *s, const int64_t *mass_ptr, const int32_t *type,
                                      const double *vec, const double *num) try {
    if (!s) return TITAN_GB300_EINVAL;
    if (s->started) return s->fail(TITAN_GB300_ESTATE, "set local constraints before start");
    if (s->n <= 0 || !mass_ptr) return s->fail(TITAN_GB300_EINVAL, "set masses first");
    int64_t nr = mass_ptr[s->n];
    if (mass_ptr[0] != 0 || nr < 0) return s->fail(TITAN_GB300_EINVAL, "bad record offsets");
    static const int order[4] = {1, 2, 0, 3};  // contact, ball, constraint plane, direction
    s->lc_ptr.assign(s->n + 1, 0);
    s->lc_type.clear();
    s->lc_rec.clear();
    for (int64_t i = 0; i < s->n; i++) {
        if (mass_ptr[i + 1] < mass_ptr[i]) return s->fail(TITAN_GB300_EINVAL, "bad record offsets");
        for (int o = 0; o < 4; o++)
            for (int64_t r = mass_ptr[i]; r < mass_ptr[i + 1]; r++) {
                if (type[r] != order[o]) continue;
                double v[3] = {vec[3 * r], vec[3 * r + 1], vec[3 * r + 2]};
                if (type[r] != TITAN_GB300_BALL) {  // constructors normalise (object.cu:60,109,127)
                    double nn = norm3(v);
                    if (nn == 0.0) return s->fail(TITAN_GB300_EINVAL, "zero constraint vector");
                    for (double &c : v) c = c / nn;
                }
                s->lc_type.push_back(type[r]);
                s->lc_rec.insert(s->lc_rec.end(), {v[0], v[1], v[2], num[r]});
            }
        s->lc_ptr[i + 1] = (int64_t)s->lc_type.size();
    }
    return TITAN_GB300_OK;
} catch (...) {
    return host_exception(s);
}

int titan_gb300_add_plane(titan_gb300_sim *s, const double normal[3], double offset, double fk, double fs) try {
    if (!s || !normal) return TITAN_GB300_EINVAL;
    if (s->serving) return s->fail(TITAN_GB300_ESTATE, "the scene is being stepped by a request server");
    if ((int)s->planes.size() >= tg::kMaxPlanes) return s->fail(TITAN_GB300_ELIMIT, "at most 16 global planes");
    double nn = norm3(normal);
    if (!(nn > 0)) return s->fail(TITAN_GB300_EINVAL, "zero plane normal");
    s->planes.push_back({normal[0] / nn, normal[1] / nn, normal[2] / nn, offset, fk, fs});
    if (s->started) return upload_params(s);
    return TITAN_GB300_OK;
} catch (...) {
    return host_exception(s);
}

int titan_gb300_add_ball(titan_gb300_sim *s, const double center[3], double radius) try {
    if (!s || !center) return TITAN_GB300_EINVAL;
    if (s->serving) return s->fail(TITAN_GB300_ESTATE, "the scene is being stepped by a request server");
    if ((int)s->balls.size() >= tg::kMaxBalls) return s->fail(TITAN_GB300_ELIMIT, "at most 16 global balls");
    s->balls.push_back({center[0], center[1], center[2], radius});
    if (s->started) return upload_params(s);
    return TITAN_GB300_OK;
} catch (...) {
    return host_exception(s);
}

int titan_gb300_clear_constraints(titan_gb300_sim *s) try {
    if (!s) return TITAN_GB300_EINVAL;
    if (s->serving) return s->fail(TITAN_GB300_ESTATE, "the scene is being stepped by a request server");
    s->planes.clear();
    s->balls.clear();
    if (s->started) return upload_params(s);
    return TITAN_GB300_OK;
} catch (...) {
    return host_exception(s);
}

int titan_gb300_set_integrator(titan_gb300_sim *s, int kind) try {
    if (!s) return TITAN_GB300_EINVAL;
    if (s->serving) return s->fail(TITAN_GB300_ESTATE, "the scene is being stepped by a request server");
    if (kind < tg::INTEG_EULER || kind > tg::INTEG_RK2)
        return s->fail(TITAN_GB300_EINVAL, "integrator must be 0 (Euler), 1 (Verlet) or 2 (RK2)");
    if (kind == s->integrator) return TITAN_GB300_OK;
    if (!s->started) {
        s->integrator = kind;
        return TITAN_GB300_OK;
    }
    if (!ensure_device(s)) return s->fail(TITAN_GB300_ECUDA, "cudaSetDevice failed");
    CK(cudaStreamSynchronize(s->stream), "set integrator");
    const bool was_res = s->use_res || s->use_rtiles;
    s->integrator = kind;
    s->dt_log.push_back({s->steps, s->dt, s->passes()});
    s->drop_graphs();
    if (was_res) {  // resident bins and tiles run Euler only: rebuild without them
        int rc = pull_state(s);
        if (rc) return rc;
        // a scene whose bodies are all above the per-step kernels' tile size
        // is resident only because it has many: its state goes over bit for
        // bit, and its accelerations (VERLET's state), as between the per-step
        // kernels
        bool carry = s->use_rtiles && !s->use_res;
        for (const tg::TileInfo &ti : s->rtiles) carry = carry && ti.nm > kWsDefaultTile && s->prec != P_FP64;
        void *rec = nullptr;
        const size_t rb = (size_t)s->n * tg::state_record_bytes(s->prec), ab = 3 * (size_t)s->n * s->rsize();
        auto xfer = [&]() {
            tg::XferArgs x{};
            x.old2new = s->d_old2new;
            x.count = s->n;
            x.npad = s->npad;
            x.state0 = s->args.state0;
            x.state1 = s->args.state1;
            x.acc = s->args.acc;
            x.parity = s->parity;
            return x;
        };
        if (carry) {
            CK(cudaMalloc(&rec, rb + ab), "carry state");
            cudaError_t e = tg::launch_carry(s->prec, xfer(), true, rec, (uint8_t *)rec + rb, s->stream);
            if (e == cudaSuccess) e = cudaStreamSynchronize(s->stream);
            if (e != cudaSuccess) {
                cudaFree(rec);
                return s->cuda_fail(e, "carry state");
            }
        }
        rc = build_device(s);
        if (carry && rc == TITAN_GB300_OK) {
            cudaError_t e = tg::launch_carry(s->prec, xfer(), false, rec, (uint8_t *)rec + rb, s->stream);
            if (e == cudaSuccess) e = cudaStreamSynchronize(s->stream);
            if (e != cudaSuccess) rc = s->cuda_fail(e, "carry state");
        }
        if (rec) cudaFree(rec);
        return rc;
    }
    // the kernels of the new integrator need their shared-memory limit
    if (s->use_pull)
        CK(tg::step_pull_prepare(s->prec, kind, (size_t)s->args.pull.total), "set shared memory");
    else if (s->use_ws)
        CK(tg::step_ws_prepare(s->prec, kind, (size_t)s->args.ws.total), "set shared memory");
    else if (!s->use_async)
        CK(tg::step_prepare(s->prec, s->step_variant, kind, s->smem), "set shared memory");
    if (int rc = prepare_grid(s)) return rc;
    return upload_params(s);
} catch (...) {
    return host_exception(s);
}

int titan_gb300_set_time_step(titan_gb300_sim *s, double dt) try {
    if (!s) return TITAN_GB300_EINVAL;
    if (s->serving) return s->fail(TITAN_GB300_ESTATE, "the scene is being stepped by a request server");
    if (!(dt > 0)) return s->fail(TITAN_GB300_EINVAL, "Cannot set time step to negative or zero value.");
    s->dt = dt;
    if (s->started) {
        s->dt_log.push_back({s->steps, dt, s->passes()});
        return upload_params(s);
    }
    return TITAN_GB300_OK;
} catch (...) {
    return host_exception(s);
}

double titan_gb300_get_time_step(const titan_gb300_sim *s) { return s ? s->dt : 0.0; }

int titan_gb300_set_global_acc(titan_gb300_sim *s, const double g[3]) try {
    if (!s || !g) return TITAN_GB300_EINVAL;
    if (s->serving) return s->fail(TITAN_GB300_ESTATE, "the scene is being stepped by a request server");
    for (int c = 0; c < 3; c++) s->g[c] = g[c];
    if (s->started) return upload_params(s);
    return TITAN_GB300_OK;
} catch (...) {
    return host_exception(s);
}

int titan_gb300_set_bodies(titan_gb300_sim *s, int64_t nbodies, const int64_t *mass_ptr) try {
    if (!s) return TITAN_GB300_EINVAL;
    s->plan_adopted = false;  // the topology may change
    if (s->started) return s->fail(TITAN_GB300_ESTATE, "set bodies before start");
    if (nbodies <= 0 || !mass_ptr || mass_ptr[0] != 0 || mass_ptr[nbodies] != s->n)
        return s->fail(TITAN_GB300_EINVAL, "body ranges must cover all masses");
    for (int64_t b = 0; b < nbodies; b++)
        if (mass_ptr[b + 1] <= mass_ptr[b]) return s->fail(TITAN_GB300_EINVAL, "empty body");
    s->body_ptr.assign(mass_ptr, mass_ptr + nbodies + 1);
    s->body_plane.assign(nbodies, {0, 0, 1, 0, 0, 0});
    s->body_has_plane.assign(nbodies, 0);
    return TITAN_GB300_OK;
} catch (...) {
    return host_exception(s);
}

int titan_gb300_set_body_plane(titan_gb300_sim *s, int64_t body, const double normal[3], double offset,
                               double fk, double fs) try {
    if (!s || !normal) return TITAN_GB300_EINVAL;
    if (s->started) return s->fail(TITAN_GB300_ESTATE, "set body planes before start");
    if (body < 0 || body >= (int64_t)s->body_plane.size()) return s->fail(TITAN_GB300_EINVAL, "no such body");
    double nn = norm3(normal);
    if (!(nn > 0)) return s->fail(TITAN_GB300_EINVAL, "zero plane normal");
    s->body_plane[body] = {normal[0] / nn, normal[1] / nn, normal[2] / nn, offset, fk, fs};
    s->body_has_plane[body] = 1;
    return TITAN_GB300_OK;
} catch (...) {
    return host_exception(s);
}

int titan_gb300_start(titan_gb300_sim *s, int tile_masses) try {
    if (!s) return TITAN_GB300_EINVAL;
    if (s->n <= 0)
        return s->fail(TITAN_GB300_EINVAL, "No masses have been added. Please add masses before starting the simulation.");
    if (!(s->dt > 0)) return s->fail(TITAN_GB300_EINVAL, "invalid time step");
    if (!ensure_device(s)) return s->fail(TITAN_GB300_ECUDA, "cudaSetDevice failed");
    if (!s->stream) CK(cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking), "create stream");
    s->tile_masses = tile_masses;
    s->T = 0.0;
    s->steps = 0;
    s->dt_log.assign(1, {0, s->dt, s->passes()});
    s->mT0.assign(s->n, 0.0);
    s->mTstep.assign(s->n, 0);
    int rc = build_device(s);
    if (rc) return rc;
    s->started = true;
    return TITAN_GB300_OK;
} catch (...) {
    return host_exception(s);
}

int titan_gb300_step(titan_gb300_sim *s, int64_t nsteps) try {
    if (!s) return TITAN_GB300_EINVAL;
    if (s->serving) return s->fail(TITAN_GB300_ESTATE, "the scene is being stepped by a request server");
    if (!s->started) return s->fail(TITAN_GB300_ESTATE, "The simulation has not started.");
    if (nsteps < 0) return s->fail(TITAN_GB300_EINVAL, "negative step count");
    if (s->torn)
        return s->fail(TITAN_GB300_ETIMEOUT, "a step kernel's wait timed out: upload all positions and velocities first");
    if (nsteps == 0) return TITAN_GB300_OK;
    if (!ensure_device(s)) return s->fail(TITAN_GB300_ECUDA, "cudaSetDevice failed");
    cudaError_t e = cudaSuccess;
    s->grid_last = 0;
    if (single_runs(s, nsteps)) {
        const int P = s->passes();
        s->gargs.T0 = s->T;
        for (int q = 0; q < P; q++) {
            CK(tg::launch_grid_single(s->prec, s->integrator, s->args, s->gargs, s->single_shape, s->grid_smem,
                                      s->parity, q, q == P - 1, s->stream, !s->tables_written),
               "launch step");
            s->tables_written = false;
            s->parity ^= 1;
            s->gargs.T0 = s->gargs.T0 + s->hprm.launch_dt;
        }
        advance_clock(s, 1);
        s->grid_last = 2;
        return TITAN_GB300_OK;
    }
    int rc_short = TITAN_GB300_OK;
    if (short_runs(s, nsteps, false, rc_short)) {
        const tg::StepArgs a = short_args(s);
        for (int64_t i = 0; i < nsteps; i++) {
            CK(tg::launch_step_ws(s->prec, s->integrator, a, s->short_form.ctas,
                                  tg::kWsMaxConsumerWarps, s->parity, i == nsteps - 1, s->stream, !s->tables_written),
               "launch step");
            s->tables_written = false;
            s->parity ^= 1;
        }
        advance_clock(s, nsteps);
        s->grid_last = 3;
        return TITAN_GB300_OK;
    }
    if (rc_short) return rc_short;
    if (grid_runs(s, nsteps)) {
        s->grid_last = 1;
        while (nsteps > 0 && s->use_grid) {
            const int64_t len = std::min(nsteps, kGridMaxSteps);
            s->gargs.T0 = s->T;
            const cudaError_t r = tg::launch_grid_resident(s->prec, s->integrator, s->args, s->gargs, s->grid_shape,
                                                           s->grid_smem, s->parity, len, 1, s->stream);
            if (r == cudaSuccess) {
                const int P = s->passes();
                s->gargs.base += (uint32_t)(len * P);
                s->parity ^= (int)((len * P) & 1);
                advance_clock(s, len);
                nsteps -= len;
                continue;
            }
            if (r != cudaErrorCooperativeLaunchTooLarge) return s->cuda_fail(r, "launch resident grid");
            cudaGetLastError();
            s->use_grid = false;  // the device has less room than planned for: per-step kernels
            s->grid_last = 0;
        }
        if (nsteps == 0) return TITAN_GB300_OK;
    }
    if (s->use_res)
        CK(tg::launch_resident(s->prec, s->args, s->rargs, s->res_ctas, s->res_threads, s->parity, nsteps, 1,
                               s->args.ntiles == 0, s->stream),
           "launch resident bins");
    const bool alone = s->args.ntiles == 0;
    if (s->use_rtiles) {
        // the first step's time: of the record's two places a step reads one and
        // writes the other, so a copy is needed only where per-step kernels
        // take more than one step beside the launch
        const double *t0 = s->args.tbuf + s->parity;
        if (!alone && nsteps > 1) {
            t0 = s->d_t0;
            CK(cudaMemcpyAsync(s->d_t0, s->args.tbuf + s->parity, sizeof(double), cudaMemcpyDeviceToDevice, s->stream),
               "launch resident tiles");
        }
        const bool own_time = alone && (nsteps & 1);
        // beside the per-step kernels and each other: disjoint masses (the
        // first group of a scene without per-step tiles needs no side stream)
        const size_t first = alone ? 1 : 0;
        if (s->rt_groups.size() > first) CK(cudaEventRecord(s->ev_fork, s->stream), "launch resident tiles");
        for (size_t q = 0; q < s->rt_groups.size(); q++) {
            const auto &g = s->rt_groups[q];
            cudaStream_t st = q < first ? s->stream : s->side_stream[q];
            if (q >= first) CK(cudaStreamWaitEvent(st, s->ev_fork, 0), "launch resident tiles");
            tg::TileResArgs r = g.args;
            r.t0 = t0;
            if (own_time && q == 0) r.time = s->args.tbuf + (s->parity ^ 1);
            CK(tg::launch_tile_resident(s->prec, s->args, r, g.mpt, g.threads, g.smem, s->parity, nsteps, 1, st),
               "launch resident tiles");
            if (q >= first) CK(cudaEventRecord(s->ev_join[q], st), "launch resident tiles");
        }
        if (alone) {
            for (size_t q = first; q < s->rt_groups.size(); q++)
                CK(cudaStreamWaitEvent(s->stream, s->ev_join[q], 0), "join resident tiles");
            if (!own_time) CK(tg::launch_advance_time(s->args, s->parity, nsteps, s->stream), "advance time");
        }
    }
    if (s->args.ntiles == 0) {
        s->parity ^= (int)(nsteps & 1);
        for (int64_t i = 0; i < nsteps; i++) s->T = s->T + s->dt;  // src/sim.cu:1590
        s->steps += nsteps;
        return TITAN_GB300_OK;
    }
    const int P = s->passes();
    const int rc = [&]() -> int {
        int64_t rem = nsteps - 1;
        while (rem > 0) {
            int len = (int)std::min<int64_t>(rem, kChunk);
            cudaGraphExec_t g = get_graph(s, len, s->parity, e);
            if (!g) return s->cuda_fail(e, "build step graph");
            CK(cudaGraphLaunch(g, s->stream), "launch step graph");
            s->tables_written = false;
            s->parity ^= ((len * P) & 1);
            rem -= len;
        }
        for (int q = 0; q < P; q++) {  // the last step also writes the accelerations
            CK(s->launch(s->parity, q == P - 1, q), "launch step");
            s->tables_written = false;
            s->parity ^= 1;
        }
        return TITAN_GB300_OK;
    }();
    // later work on the handle's stream sees the resident tiles' results
    if (s->use_rtiles)
        for (size_t q = 0; q < s->rt_groups.size(); q++)
            CK(cudaStreamWaitEvent(s->stream, s->ev_join[q], 0), "join resident tiles");
    if (rc) return rc;
    advance_clock(s, nsteps);
    return TITAN_GB300_OK;
} catch (...) {
    return host_exception(s);
}

int titan_gb300_prepare_steps(titan_gb300_sim *s, int64_t nsteps) try {
    if (!s) return TITAN_GB300_EINVAL;
    if (s->serving) return s->fail(TITAN_GB300_ESTATE, "the scene is being stepped by a request server");
    if (!s->started) return s->fail(TITAN_GB300_ESTATE, "The simulation has not started.");
    if (nsteps < 0) return s->fail(TITAN_GB300_EINVAL, "negative step count");
    if (!ensure_device(s)) return s->fail(TITAN_GB300_ECUDA, "cudaSetDevice failed");
    if (int rc = TITAN_GB300_OK; nsteps > 0 && (short_runs(s, nsteps, true, rc) || rc)) return rc;
    if (s->args.ntiles == 0 || nsteps <= 1 || grid_runs(s, nsteps)) return TITAN_GB300_OK;
    // the same chunk sequence step(nsteps) replays, from the current parity
    cudaError_t e = cudaSuccess;
    const int P = s->passes();
    int parity = s->parity;
    for (int64_t rem = nsteps - 1; rem > 0;) {
        const int len = (int)std::min<int64_t>(rem, kChunk);
        if (!get_graph(s, len, parity, e)) return s->cuda_fail(e, "build step graph");
        parity ^= ((len * P) & 1);
        rem -= len;
    }
    return TITAN_GB300_OK;
} catch (...) {
    return host_exception(s);
}

int titan_gb300_synchronize(titan_gb300_sim *s) try {
    if (!s) return TITAN_GB300_EINVAL;
    if (!s->stream) return TITAN_GB300_OK;
    CK(cudaStreamSynchronize(s->stream), "synchronize");
    return check_kernel_error(s);
} catch (...) {
    return host_exception(s);
}

int titan_gb300_poll(titan_gb300_sim *s) try {
    if (!s) return TITAN_GB300_EINVAL;
    if (!s->stream) return TITAN_GB300_OK;
    if (!ensure_device(s)) return s->fail(TITAN_GB300_ECUDA, "cudaSetDevice failed");
    const cudaError_t e = cudaStreamQuery(s->stream);
    if (e == cudaErrorNotReady) return TITAN_GB300_EBUSY;
    if (e != cudaSuccess) return s->cuda_fail(e, "poll");
    return check_kernel_error(s);
} catch (...) {
    return host_exception(s);
}

int titan_gb300_wait(titan_gb300_sim *s, double timeout_ms) try {
    if (!s) return TITAN_GB300_EINVAL;
    if (!(timeout_ms >= 0)) return s->fail(TITAN_GB300_EINVAL, "timeout must be >= 0");
    const auto t0 = std::chrono::steady_clock::now();
    for (;;) {
        const int rc = titan_gb300_poll(s);
        if (rc != TITAN_GB300_EBUSY) return rc;
        const double ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
        if (ms >= timeout_ms) return s->fail(TITAN_GB300_ETIMEOUT, "queued steps still running at the time limit");
        std::this_thread::sleep_for(std::chrono::microseconds(50));
    }
} catch (...) {
    return host_exception(s);
}

int titan_gb300_export_vertices(titan_gb300_sim *s, float *out, int out_on_device) try {
    if (!s || !out) return TITAN_GB300_EINVAL;
    if (s->serving) return s->fail(TITAN_GB300_ESTATE, "the scene is being stepped by a request server");
    if (!s->started) return s->fail(TITAN_GB300_ESTATE, "The simulation has not started.");
    if (!ensure_device(s)) return s->fail(TITAN_GB300_ECUDA, "cudaSetDevice failed");
    tg::XferArgs x{};
    x.old2new = s->d_old2new;
    x.count = s->n;
    x.npad = s->npad;
    x.state0 = s->args.state0;
    x.state1 = s->args.state1;
    x.acc = s->args.acc;
    x.parity = s->parity;
    if (out_on_device) {
        CK(tg::launch_export_f32(s->prec, x, out, s->stream), "export vertices");
        return TITAN_GB300_OK;
    }
    // host buffer: through the staging area (9n doubles >= 3n floats)
    float *d = reinterpret_cast<float *>(s->d_xfer);
    CK(tg::launch_export_f32(s->prec, x, d, s->stream), "export vertices");
    CK(cudaMemcpyAsync(out, d, 3 * (size_t)s->n * sizeof(float), cudaMemcpyDeviceToHost, s->stream),
       "export vertices");
    CK(cudaStreamSynchronize(s->stream), "export vertices");
    return TITAN_GB300_OK;
} catch (...) {
    return host_exception(s);
}

int titan_gb300_export_indices(titan_gb300_sim *s, uint32_t *out, int out_on_device) try {
    if (!s || !out) return TITAN_GB300_EINVAL;
    if (s->serving) return s->fail(TITAN_GB300_ESTATE, "the scene is being stepped by a request server");
    std::vector<uint32_t> idx(2 * (size_t)s->ns, 0);
    for (int64_t j = 0; j < s->ns; j++) {
        const int32_t l = s->left[j], r = s->right[j];
        if (l < 0 || r < 0 || l >= s->n || r >= s->n) continue;  // detached: (0, 0)
        idx[2 * j] = (uint32_t)l;
        idx[2 * j + 1] = (uint32_t)r;
    }
    if (!out_on_device) {
        if (!idx.empty()) std::memcpy(out, idx.data(), idx.size() * sizeof(uint32_t));
        return TITAN_GB300_OK;
    }
    if (!s->started) return s->fail(TITAN_GB300_ESTATE, "The simulation has not started.");
    if (!ensure_device(s)) return s->fail(TITAN_GB300_ECUDA, "cudaSetDevice failed");
    if (!idx.empty())
        CK(cudaMemcpy(out, idx.data(), idx.size() * sizeof(uint32_t), cudaMemcpyHostToDevice), "export indices");
    return TITAN_GB300_OK;
} catch (...) {
    return host_exception(s);
}

double titan_gb300_time(const titan_gb300_sim *s) { return s ? s->T : 0.0; }

int64_t titan_gb300_device_bytes(const titan_gb300_sim *s) {
    return s ? (int64_t)(s->mem.total + spring_update_bytes(s)) : 0;
}

void *titan_gb300_host_alloc(size_t bytes) {
    void *p = nullptr;
    if (bytes == 0 || cudaMallocHost(&p, bytes) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return p;
}

void titan_gb300_host_free(void *p) {
    if (p) cudaFreeHost(p);
}

int titan_gb300_set_time(titan_gb300_sim *s, double T) try {
    if (!s) return TITAN_GB300_EINVAL;
    if (s->serving) return s->fail(TITAN_GB300_ESTATE, "the scene is being stepped by a request server");
    s->T = T;
    if (!s->started) return TITAN_GB300_OK;
    if (!ensure_device(s)) return s->fail(TITAN_GB300_ECUDA, "cudaSetDevice failed");
    return upload_params(s);
} catch (...) {
    return host_exception(s);
}
int64_t titan_gb300_steps(const titan_gb300_sim *s) { return s ? s->steps : 0; }

int titan_gb300_get_masses(titan_gb300_sim *s, int64_t count, const int64_t *idx, double *pos, double *vel,
                           double *acc, double *T) try {
    if (!s) return TITAN_GB300_EINVAL;
    if (s->serving) return s->fail(TITAN_GB300_ESTATE, "the scene is being stepped by a request server");
    if (!s->started) return s->fail(TITAN_GB300_ESTATE, "The simulation has not started.");
    if (count < 0 || count > s->n) return s->fail(TITAN_GB300_EINVAL, "bad count");
    if (idx)
        for (int64_t q = 0; q < count; q++)
            if (idx[q] < 0 || idx[q] >= s->n) return s->fail(TITAN_GB300_EINVAL, "mass index out of range");
    if (count == 0) return TITAN_GB300_OK;
    if (!ensure_device(s)) return s->fail(TITAN_GB300_ECUDA, "cudaSetDevice failed");
    tg::XferArgs x{};
    x.old2new = s->d_old2new;
    x.count = count;
    x.npad = s->npad;
    x.state0 = s->args.state0;
    x.state1 = s->args.state1;
    x.acc = s->args.acc;
    x.parity = s->parity;
    if (idx) {
        CK(cudaMemcpyAsync(s->d_idx, idx, count * 8, cudaMemcpyHostToDevice, s->stream), "upload index");
        x.idx = s->d_idx;
    }
    // only the requested arrays come back: the kernel writes them into a
    // caller buffer that is page-locked as a whole, else into the handle's
    // staging buffer, and the error flag beside that
    double *outs[3] = {pos, vel, acc}, *dst[3] = {nullptr, nullptr, nullptr};
    bool direct[3] = {false, false, false};
    const bool any = pos || vel || acc;
    if (any) {
        for (int q = 0; q < 3; q++) {
            if (!outs[q]) continue;
            double *const h = (double *)host_on_device(outs[q], 3 * (size_t)count * 8);
            direct[q] = h && (reinterpret_cast<uintptr_t>(h) & 7) == 0;
            dst[q] = direct[q] ? h : s->stage_dev + 3 * q * count;
        }
        x.pos = dst[0];
        x.vel = dst[1];
        x.accout = dst[2];
        x.err = s->d_err;
        x.err_out = reinterpret_cast<int *>(s->stage_dev + 9 * s->n);
        CK(tg::launch_gather(s->prec, x, s->stream), "gather");
    }
    CK(cudaStreamSynchronize(s->stream), "download");
    if (!any || *s->h_err)
        if (int rc = check_kernel_error(s)) return rc;
    for (int q = 0; q < 3; q++)
        if (outs[q] && !direct[q]) par_memcpy(outs[q], s->h_xfer + 3 * q * count, 3 * count * 8);
    if (T) mass_times(s, idx, count, T);
    return TITAN_GB300_OK;
} catch (...) {
    return host_exception(s);
}

int titan_gb300_get_state(titan_gb300_sim *s, double *pos, double *vel, double *acc, double *T) try {
    if (!s) return TITAN_GB300_EINVAL;
    if (s->serving) return s->fail(TITAN_GB300_ESTATE, "the scene is being stepped by a request server");
    return titan_gb300_get_masses(s, s->n, nullptr, pos, vel, acc, T);
} catch (...) {
    return host_exception(s);
}

int titan_gb300_set_mass_state(titan_gb300_sim *s, int64_t count, const int64_t *idx, const double *pos,
                               const double *vel, const double *m, const double *ext, const uint8_t *fixed,
                               const double *drag, const double *T) try {
    if (!s) return TITAN_GB300_EINVAL;
    if (s->serving) return s->fail(TITAN_GB300_ESTATE, "the scene is being stepped by a request server");
    if (!s->started) return s->fail(TITAN_GB300_ESTATE, "The simulation has not started.");
    if (!idx) count = s->n;
    if (count < 0 || count > s->n) return s->fail(TITAN_GB300_EINVAL, "bad count");
    for (int64_t q = 0; idx && q < count; q++)
        if (idx[q] < 0 || idx[q] >= s->n) return s->fail(TITAN_GB300_EINVAL, "mass index out of range");
    if (m)
        for (int64_t q = 0; q < count; q++)
            if (!(m[q] > 0)) return s->fail(TITAN_GB300_EINVAL, "mass must be positive");
    if (!ensure_device(s)) return s->fail(TITAN_GB300_ECUDA, "cudaSetDevice failed");
    CK(cudaStreamSynchronize(s->stream), "set");
    bool replan = false;
    if (fixed) {
        if (s->fixed.empty()) s->fixed.assign(s->n, 0);
        for (int64_t q = 0; q < count; q++) {
            int64_t i = idx ? idx[q] : q;
            if ((s->fixed[i] != 0) != (fixed[q] != 0)) replan = true;
        }
    }
    // local time bookkeeping: masses whose T is given, or whose fixed flag
    // flips, restart their clock here
    std::vector<double> Tcur;
    if (replan || T) {
        Tcur.resize(s->n);
        mass_times(s, nullptr, s->n, Tcur.data());
    }
    // per-mass host bookkeeping, only for the attributes given (a loop over
    // every mass costs milliseconds on a million-mass scene)
    for (int64_t q = 0; (m || ext || drag || T || fixed) && q < count; q++) {
        int64_t i = idx ? idx[q] : q;
        if (m) s->m[i] = m[q];
        if (ext) {
            if (s->ext.empty()) s->ext.assign(3 * s->n, 0.0);
            for (int c = 0; c < 3; c++) s->ext[3 * i + c] = ext[3 * q + c];
        }
        if (drag) {
            if (s->drag.empty()) s->drag.assign(s->n, 0);
            s->drag[i] = (int32_t)drag[q];
        }
        if (T || (fixed && (s->fixed[i] != 0) != (fixed[q] != 0))) {
            s->mT0[i] = T ? T[q] : Tcur[i];
            s->mTstep[i] = s->steps;
        }
        if (fixed) s->fixed[i] = fixed[q] ? 1 : 0;
    }
    if (replan) {
        int rc = pull_state(s);
        if (rc) return rc;
        for (int64_t q = 0; q < count; q++) {
            int64_t i = idx ? idx[q] : q;
            for (int c = 0; c < 3; c++) {
                if (pos) s->pos[3 * i + c] = pos[3 * q + c];
                if (vel) s->vel[3 * i + c] = vel[3 * q + c];
            }
        }
        s->drop_graphs();
        return build_device(s);
    }
    if (m || ext || drag) {
        int rc = upload_mass_attrs(s);
        if (rc) return rc;
    }
    if (pos || vel) {
        tg::XferArgs x{};
        x.old2new = s->d_old2new;
        x.count = count;
        x.npad = s->npad;
        x.state0 = s->args.state0;
        x.state1 = s->args.state1;
        x.acc = s->args.acc;
        x.parity = s->parity;
        if (idx) {
            CK(cudaMemcpyAsync(s->d_idx, idx, count * 8, cudaMemcpyHostToDevice, s->stream), "upload index");
            x.idx = s->d_idx;
        }
        // a pinned caller buffer goes up by DMA directly, else through the
        // handle's pinned staging buffer
        const double *ins[2] = {pos, vel};
        for (int q = 0; q < 2; q++) {
            if (!ins[q]) continue;
            const double *src = ins[q];
            if (!host_pinned(src)) {
                par_memcpy(s->h_xfer + 3 * q * count, src, 3 * count * 8);
                src = s->h_xfer + 3 * q * count;
            }
            CK(cudaMemcpyAsync(s->d_xfer + 3 * q * count, src, 3 * count * 8, cudaMemcpyHostToDevice, s->stream),
               "upload");
        }
        x.ipos = pos ? s->d_xfer : nullptr;
        x.ivel = vel ? s->d_xfer + 3 * count : nullptr;
        CK(tg::launch_scatter(s->prec, x, s->stream), "scatter");
        CK(cudaStreamSynchronize(s->stream), "set");
        if (s->torn && !idx && pos && vel) {  // a whole state again; the time record, too
            if (int rc = upload_params(s)) return rc;
            s->torn = false;
        }
    }
    return TITAN_GB300_OK;
} catch (...) {
    return host_exception(s);
}

int titan_gb300_set_spring_params(titan_gb300_sim *s, int64_t count, const int64_t *idx, const double *k,
                                  const double *rest, const double *damping, const int32_t *type,
                                  const double *omega, const double *amp, const double *phase) try {
    if (!s) return TITAN_GB300_EINVAL;
    if (s->serving) return s->fail(TITAN_GB300_ESTATE, "the scene is being stepped by a request server");
    if (!idx) count = s->ns;
    if (count < 0 || count > s->ns) return s->fail(TITAN_GB300_EINVAL, "bad count");
    bool replan = false;
    for (int64_t q = 0; q < count; q++) {
        int64_t j = idx ? idx[q] : q;
        if (j < 0 || j >= s->ns) return s->fail(TITAN_GB300_EINVAL, "spring index out of range");
        if (type && (type[q] < 0 || type[q] > 3)) return s->fail(TITAN_GB300_EINVAL, "spring type must be 0..3");
    }
    if (s->started) {  // what the stream still has to do reads the host arrays
        if (!ensure_device(s)) return s->fail(TITAN_GB300_ECUDA, "cudaSetDevice failed");
        CK(cudaStreamSynchronize(s->stream), "set springs");
    }
    if (omega && s->omega.empty()) s->omega.assign(s->ns, 0.0);
    if (amp && s->amp.empty()) s->amp.assign(s->ns, 0.2);
    if (phase && s->phase.empty()) s->phase.assign(s->ns, 0.0);
    const double *in[] = {k, rest, damping, omega, amp, phase};
    std::vector<double> *host[] = {&s->k, &s->rest, &s->damping, &s->omega, &s->amp, &s->phase};
    unsigned given = 0;
    for (int q = 0; q < titan_gb300_sim::SP_COUNT; q++) {
        if (!in[q] || count == 0) continue;
        given |= 1u << q;
        s->sp_current[q] = false;
        if (idx)
            for (int64_t i = 0; i < count; i++) (*host[q])[idx[i]] = in[q][i];
        else
            par_memcpy(host[q]->data(), in[q], count * 8);
    }
    bool retyped = false;
    if (type) {
        if (s->type.empty()) s->type.assign(s->ns, 0);
        for (int64_t q = 0; q < count; q++) {
            int64_t j = idx ? idx[q] : q;
            bool was = s->type[j] >= 2, now = type[q] >= 2;
            if (was != now) replan = true;
            retyped |= s->type[j] != type[q];
            s->type[j] = type[q];
        }
    }
    if (!s->started) return TITAN_GB300_OK;
    if (replan) {
        int rc = pull_state(s);
        if (rc) return rc;
        s->drop_graphs();
        return build_device(s);
    }
    if (!given && !retyped) return TITAN_GB300_OK;
    // no new types: the device rewrites the slab records
    if (!retyped && !s->use_res && !s->use_pull) {
        bool done = false;
        const int rc = refresh_entries(s, given, done);
        if (rc || done) return rc;
    }
    // type changes within passive or within active keep the slab order, but
    // the type bits live in the entry words
    if (type) {
        for (size_t e = 0; e < s->plan.ent_ends.size(); e++) {
            int64_t j = s->plan.ent_spring[e];
            s->plan.ent_ends[e] = (s->plan.ent_ends[e] & 0x00ffffffu) | ((uint32_t)(s->type[j] & 3) << 24);
        }
        if (s->use_res)
            for (size_t q = 0; q < s->rplan.words.size(); q++) {
                int64_t j = s->rplan.rec_spring[q];
                if (j >= 0) s->rplan.words[q] = (s->rplan.words[q] & 0xffffu) | ((uint32_t)(s->type[j] & 3) << 16);
            }
    }
    return upload_entries(s);
} catch (...) {
    return host_exception(s);
}

int titan_gb300_diagnostics(titan_gb300_sim *s, double g_mag, double energy[4], double momentum[6]) try {
    if (!s) return TITAN_GB300_EINVAL;
    if (s->serving) return s->fail(TITAN_GB300_ESTATE, "the scene is being stepped by a request server");
    if (!s->started) return s->fail(TITAN_GB300_ESTATE, "The simulation has not started.");
    if (!ensure_device(s)) return s->fail(TITAN_GB300_ECUDA, "cudaSetDevice failed");
    cudaError_t e = cudaSuccess;
    if (!s->d_sl) {
        std::vector<int32_t> sl(s->ns, -1), sr(s->ns, -1);
        for (int64_t j = 0; j < s->ns; j++) {
            int32_t l = s->left[j], r = s->right[j];
            if (l < 0 || r < 0 || l >= s->n || r >= s->n) continue;
            sl[j] = s->plan.old2new[l];
            sr[j] = s->plan.old2new[r];
        }
        if (!(s->d_sl = dev_copy(s, sl, e))) return s->cuda_fail(e, "diag alloc");
        if (!(s->d_sr = dev_copy(s, sr, e))) return s->cuda_fail(e, "diag alloc");
        if (!(s->d_partials = (double *)s->mem.get(tg::kDiagBlocks * tg::kDiagQ * 8, e)))
            return s->cuda_fail(e, "diag alloc");
        if (!(s->d_dout = (double *)s->mem.get(tg::kDiagQ * 8, e))) return s->cuda_fail(e, "diag alloc");
    }
    // (the host arrays change only after a wait for this stream)
    constexpr unsigned kLengths = 1u << titan_gb300_sim::SP_K | 1u << titan_gb300_sim::SP_REST;
    if (!alloc_spring_arrays(s, kLengths, e)) return s->cuda_fail(e, "diag alloc");
    if (int rc = upload_spring_arrays(s, kLengths)) return rc;
    tg::DiagArgs d{};
    d.state = s->parity ? s->args.state1 : s->args.state0;
    d.mass = s->args.mass;
    d.n = s->n;
    d.npad = s->npad;
    d.sl = s->d_sl;
    d.sr = s->d_sr;
    d.sk = s->d_sp[titan_gb300_sim::SP_K];
    d.srest = s->d_sp[titan_gb300_sim::SP_REST];
    d.ns = s->ns;
    d.g_mag = g_mag;
    d.partials = s->d_partials;
    d.out = s->d_dout;
    CK(tg::launch_diag(s->prec, d, s->stream), "diagnostics");
    double out[tg::kDiagQ];
    CK(cudaMemcpyAsync(out, s->d_dout, sizeof(out), cudaMemcpyDeviceToHost, s->stream), "diag download");
    CK(cudaStreamSynchronize(s->stream), "diagnostics");
    if (energy) {
        energy[0] = out[0];
        energy[1] = out[1];
        energy[2] = out[2];
        energy[3] = (out[0] + out[1]) + out[2];
    }
    if (momentum)
        for (int c = 0; c < 6; c++) momentum[c] = out[3 + c];
    return TITAN_GB300_OK;
} catch (...) {
    return host_exception(s);
}

void *titan_gb300_stream(titan_gb300_sim *s) { return s ? (void *)s->stream : nullptr; }

int titan_gb300_plan_info(const titan_gb300_sim *s, int64_t out[12]) {
    if (!s || !out) return TITAN_GB300_EINVAL;
    const tg::Plan &P = s->plan;
    std::memset(out, 0, 12 * sizeof(int64_t));
    out[0] = s->n;
    out[1] = s->ns;
    if (!s->started) return TITAN_GB300_OK;
    out[2] = P.ntiles;
    out[3] = (int64_t)P.ent_ends.size();
    out[4] = (int64_t)P.halo.size();
    out[5] = (int64_t)P.inc.size();
    out[6] = (int64_t)P.heavy_local.size();
    out[7] = (int64_t)s->smem;
    out[8] = s->threads;
    int64_t nact_springs = 0;
    if (!s->type.empty())
        for (int32_t t : s->type) nact_springs += t >= 2;
    int64_t nact_ent = 0;
    for (int32_t a : P.tile_nact) nact_ent += a;
    const bool f64 = s->prec == P_FP64;
    // algorithmic bytes per step: per mass read x,v,m,flags + write x,v;
    // per spring k, rest, damping + two endpoint indices; actuated springs
    // add omega and phase.
    int64_t mass_b = f64 ? 105 : (s->prec == P_FP32C ? 101 : 53);
    int64_t spring_b = f64 ? 32 : 20, act_b = f64 ? 16 : 8;
    out[9] = s->n * mass_b + P.valid_springs * spring_b + nact_springs * act_b;
    // implementation bytes as laid out: per mass state read (+halo re-reads)
    // and write, m, flags, degree; per entry record, act record, 2 B per
    // incidence word, 4 B per halo index, tile table.
    const int64_t rs = (int64_t)s->rsize();
    const int64_t comps = s->comps();
    int64_t impl = s->n * (comps * rs * 2 + rs + 1 + 1) + (int64_t)P.halo.size() * (f64 ? 48 : 36);
    impl += (int64_t)P.ent_ends.size() * (f64 ? 32 : 16) + nact_ent * (f64 ? 32 : 16);
    impl += (int64_t)P.inc.size() * 2 + (int64_t)P.heavy_inc.size() * 2 + (int64_t)P.halo.size() * 4;
    impl += P.ntiles * (int64_t)sizeof(tg::TileInfo);
    out[10] = s->use_pull ? s->pull_impl_bytes : impl;
    out[11] = nact_ent;
    return TITAN_GB300_OK;
}

int64_t titan_gb300_lattice_springs(int nx, int ny, int nz);

}  // extern "C"
