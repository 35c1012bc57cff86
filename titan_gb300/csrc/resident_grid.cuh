// resident_grid.cuh -- every tile of a scene on its own CTA, all steps of a
// call in one cooperative launch (calls above 512 steps in several).
//
// The per-step kernels pay, for every step, a launch, the staging of each
// tile's state and slab, and the drain at the grid's end; on a scene whose
// tiles all fit the GPU at once that is most of the step.  Here each CTA
// keeps its tile's state records in shared memory (and, when they fit, its
// slab, actuation and incidence records) and only the halo moves.  After a
// pass a CTA writes the new records of the masses that other tiles read to an
// exchange buffer, as 16-byte chunks of three words and the number of the
// pass, and a reader polls each chunk until that number is there: no fence,
// flag or barrier stands between the tiles (with counts published behind a
// fence and polled per tile a pass took 1.1 us more).
//
// Two exchange buffers are enough.  A tile overwrites its pass k records in
// pass k + 2, after it has read the pass k + 1 records of its halo; the tile
// that wrote one of those had read the pass k records it needed.  Every tile
// that reads a free mass of this one does so for a spring between two free
// masses, which is in this tile's slab too, with the other end in its halo;
// fixed masses are neither written nor waited for.
//
// Measured, us per step, with the per-step kernels and here: FP64 5^3 8.6 ->
// 4.6, 9^3 12.7 -> 6.2, 20^3 16.1 -> 12.3, 24^3 22.4 -> 17.4, 30^3 32.2 -> 28.0,
// 96 bodies of 3-9 masses per side 38.6 -> 27.0; FP32C 9^3 4.0 -> 2.6, 16^3 4.1
// -> 2.7, 23^3 5.6 -> 3.9, 30^3 7.9 -> 5.7, 37^3 11.8 -> 8.1.  The exchange is
// about 0.7 us of a step; the rest is the latency of one tile's phases (20^3
// FP64: FP64 pipe 46 % busy, 1.55 instructions per clock; 23^3 FP32C: 1.43).
//
// The phases and the order of every sum are the per-step kernels'
// (tile_phases.cuh, epilogue.cuh): the results are the same bits.  Waits are
// bounded: a CTA that gives up raises *err, which the others poll.  The
// launch is cooperative, so all CTAs run at once.
//
// A single step has no exchange, so its launch need not be cooperative: in
// the FP32 forms it is one pass with programmatic stream serialisation, whose
// CTAs stage their tables while the step before drains (launch_grid_single).
// The tiles cut for this kernel are small for the warp-specialised one.  us
// per step(1), FP32C, that kernel and this: 12^3 4.3 and 3.9, 16^3 5.3 and 4.2,
// 20^3 5.8 and 4.7, 23^3 6.0 and 5.3, 26^3 6.5 and 5.9, 30^3 7.0 and 7.8 (there,
// above 64 masses a tile, it is not used); with that kernel and its own larger
// tiles 4.2, 4.2, 5.0, 5.5, 6.2 and 7.8.
#pragma once

#include <cstdint>

#include "engine.h"
#include "epilogue.cuh"
#include "epilogue_lanes.cuh"
#include "grid_dep.cuh"
#include "state.cuh"
#include "step_math.cuh"
#include "tile_phases.cuh"

namespace tg {

namespace {

// launch shapes: threads per CTA and CTAs per SM, at most 128 registers each
struct GridShape {
    int threads, ctas;
};
constexpr GridShape kShapes[kGridShapes] = {{512, 1}, {256, 2}, {128, 4}};
constexpr int kLaneWarps = 8;  // warps a tile's masses may take with a lane per component

__host__ __device__ constexpr int64_t rg_align16(int64_t x) { return (x + 15) & ~int64_t(15); }
constexpr int64_t kParamBytes = (int64_t)sizeof(DevParams);  // a multiple of 16

// Byte offsets of one tile's shared-memory regions.
struct RgLayout {
    int64_t st, slots, heavy, sum, ent, act, inc, total;
};
__host__ __device__ inline RgLayout rg_layout(int precision, const TileInfo &ti, int stage) {
    const int64_t rec = precision == P_FP32 ? 32 : 48, slot = precision == P_FP64 ? 32 : 16;
    RgLayout L;
    L.st = kParamBytes;
    L.slots = L.st + rg_align16((int64_t)(ti.nm + ti.nh) * rec);
    L.heavy = L.slots + ((int64_t)ti.ne + 1) * slot;  // + the zero slot padding codes name
    L.sum = L.heavy + rg_align16(3 * (int64_t)ti.nheavy * (precision == P_FP64 ? 8 : 4));
    L.ent = L.sum + (precision == P_FP64 ? rg_align16(24 * (int64_t)ti.nm) : 0);
    L.act = L.ent + (stage ? (int64_t)ti.ne * slot : 0);
    L.inc = L.act + (stage ? (int64_t)ti.nact * slot : 0);
    L.total = L.inc + (stage ? rg_align16((int64_t)ti.inc_words * 2) : 0);
    return L;
}

// One chunk of the exchange buffer: 128-bit loads and stores that are single
// accesses, through L2.
struct Chunk {
    uint32_t w[3], tag;
};
__device__ __forceinline__ Chunk ld_chunk(const void *p) {
    uint64_t lo, hi;
    asm volatile("{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}"
                 : "=l"(lo), "=l"(hi)
                 : "l"(p)
                 : "memory");
    return Chunk{{(uint32_t)lo, (uint32_t)(lo >> 32), (uint32_t)hi}, (uint32_t)(hi >> 32)};
}
__device__ __forceinline__ void st_chunk(void *p, const Chunk &c) {
    const uint64_t lo = ((uint64_t)c.w[1] << 32) | c.w[0], hi = ((uint64_t)c.tag << 32) | c.w[2];
    asm volatile("{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}" ::"l"(p), "l"(lo),
                 "l"(hi)
                 : "memory");
}

// Data that the step before wrote.  In the FP32 forms around L1 and the
// read-only path: a single step starts while that step still writes.
template <int PREC, class T>
__device__ __forceinline__ T load_fresh(const T *p) {
    if constexpr (PREC == P_FP64) return __ldg(p);
    else return __ldcg(p);
}

// The words of a state record that the exchange carries.
template <int PREC>
__device__ __forceinline__ void record_words(const St<PREC> &s, uint32_t *w) {
    if constexpr (PREC == P_FP64) {
#pragma unroll
        for (int c = 0; c < 3; c++) {
            w[2 * c] = (uint32_t)__double2loint(s.x[c]);
            w[2 * c + 1] = (uint32_t)__double2hiint(s.x[c]);
            w[6 + 2 * c] = (uint32_t)__double2loint(s.v[c]);
            w[7 + 2 * c] = (uint32_t)__double2hiint(s.v[c]);
        }
    } else {
#pragma unroll
        for (int c = 0; c < 3; c++) {
            w[c] = __float_as_uint(s.x[c]);
            w[3 + c] = __float_as_uint(s.v[c]);
            if constexpr (PREC == P_FP32C) {
                w[6 + c] = __float_as_uint(s.xl[c]);
                w[9 + c] = __float_as_uint(s.vl[c]);
            }
        }
    }
}

template <int PREC, int INTEG, int STAGE, int SHAPE, bool LANES>
__global__ void __launch_bounds__(kShapes[SHAPE].threads, kShapes[SHAPE].ctas)
    k_grid_resident(StepArgs a, GridResArgs r, int parity, int64_t passes, int write_acc) {
    using R = typename Real<PREC>::T;
    constexpr int kRec = PREC == P_FP32 ? 32 : 48;
    constexpr int kSlot = Slot<PREC>::kBytes;
    constexpr int kBatch = PREC == P_FP64 ? 1 : 3;  // slab entries a thread has in flight (measured best)
    constexpr int kChunks = PREC == P_FP32 ? 2 : 4;  // of one record in the exchange
    constexpr int kPoll = 4;                         // chunks a thread has in flight
    extern __shared__ __align__(16) uint8_t smem[];
    const DevParams *prm = reinterpret_cast<const DevParams *>(smem);
    for (int v = threadIdx.x; v < (int)(kParamBytes / 16); v += blockDim.x)
        reinterpret_cast<float4 *>(smem)[v] = __ldg(reinterpret_cast<const float4 *>(a.prm) + v);
    const TileInfo ti = r.tiles[blockIdx.x];
    const int nm = ti.nm, nh = ti.nh, E = ti.ne;
    const RgLayout L = rg_layout(PREC, ti, STAGE);
    uint8_t *const st = smem + L.st;
    uint8_t *const slots = smem + L.slots;
    R *const sH = reinterpret_cast<R *>(smem + L.heavy);
    double *const sF = reinterpret_cast<double *>(smem + L.sum);
    const uint8_t *gent = reinterpret_cast<const uint8_t *>(a.ent) + (int64_t)ti.ent_off * kSlot;
    const uint8_t *gact = reinterpret_cast<const uint8_t *>(a.act) + (int64_t)ti.ent_off * kSlot;
    const uint16_t *incb = STAGE ? reinterpret_cast<const uint16_t *>(smem + L.inc) : a.inc;
    const uint32_t inc_base = STAGE ? (uint32_t)ti.inc_off : 0u;
    const int64_t np = a.npad;

    // the tile's state and tables; no step writes the tables, so a single step
    // stages them before it waits for the one before
    constexpr int kVec = kRec / 16;
    auto load_tile = [&]() {
        const float4 *src = reinterpret_cast<const float4 *>(
            reinterpret_cast<const uint8_t *>(parity ? a.state1 : a.state0) + (int64_t)ti.mass_off * kRec);
        for (int v = threadIdx.x; v < nm * kVec; v += blockDim.x)
            reinterpret_cast<float4 *>(st)[v] = load_fresh<PREC>(src + v);
    };
    const bool single = PREC != P_FP64 && r.single;
    if constexpr (PREC == P_FP64) load_tile();
    if (single) grid_dep_launch_dependents();
    if constexpr (STAGE) {
        for (int v = threadIdx.x; v < E * (kSlot / 16); v += blockDim.x)
            reinterpret_cast<float4 *>(smem + L.ent)[v] = __ldg(reinterpret_cast<const float4 *>(gent) + v);
        for (int v = threadIdx.x; v < ti.nact * (kSlot / 16); v += blockDim.x)
            reinterpret_cast<float4 *>(smem + L.act)[v] = __ldg(reinterpret_cast<const float4 *>(gact) + v);
        const uint2 *gi = reinterpret_cast<const uint2 *>(a.inc + ti.inc_off);
        for (int v = threadIdx.x; v < ti.inc_words / 4; v += blockDim.x)
            reinterpret_cast<uint2 *>(smem + L.inc)[v] = __ldg(gi + v);
    }
    if (threadIdx.x < kSlot / 16)
        reinterpret_cast<float4 *>(slots + (int64_t)E * kSlot)[threadIdx.x] = make_float4(0.f, 0.f, 0.f, 0.f);

    // this thread's own mass (a tile has at most blockDim.x masses)
    const int i_own = threadIdx.x;
    const int64_t g_own = (int64_t)ti.mass_off + i_own;
    uint8_t fl = MF_FIXED;
    uint32_t d = 0, woff = 0;
    R m = 1;
    if (i_own < nm) {
        fl = __ldg(a.flags + g_own);
        d = __ldg(a.deg + g_own);
        m = __ldg(reinterpret_cast<const R *>(a.mass) + g_own);
        woff = __ldg(a.warp_inc_off + ti.warp_off + (i_own >> 5)) - inc_base;
    }
    // FP64: the sum of component c of mass ic, in the thread that has it: on
    // small tiles a lane per component for the whole mass phase
    // (epilogue_lanes.cuh), else whole warps per component where there is a
    // thread for each (step_kernel.cuh)
    const int nmp = (nm + 31) & ~31;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool split = PREC == P_FP64 && (LANES || 3 * nmp <= (int)blockDim.x);
    const int c_sp = LANES ? min(lane / kLaneMasses, 2)
                           : ((int)threadIdx.x >= 2 * nmp ? 2 : ((int)threadIdx.x >= nmp ? 1 : 0));
    const int i_sp = !LANES ? (int)threadIdx.x - c_sp * nmp
                            : lane < 3 * kLaneMasses ? warp * kLaneMasses + lane % kLaneMasses : nm;
    uint32_t d_sp = 0, woff_sp = 0;
    if (split && i_sp < nm) {
        d_sp = __ldg(a.deg + ti.mass_off + i_sp);
        if (d_sp == 255) d_sp = LANES ? 255 : 0;
        woff_sp = __ldg(a.warp_inc_off + ti.warp_off + (i_sp >> 5)) - inc_base;
    }

    // the thread's incidence words
    const uint32_t d_c = split ? (d_sp == 255 ? 0 : d_sp) : (d == 255 ? 0 : d), nw = (d_c + 3) >> 2, pad = (uint32_t)E * 0x10001u;
    const uint2 *const ip = reinterpret_cast<const uint2 *>(incb + (split ? woff_sp : woff)) +
                            ((split ? i_sp : i_own) & 31);
    auto word = [&](uint32_t w) { return w >= nw ? make_uint2(pad, pad) : STAGE ? ip[32 * w] : __ldg(ip + 32 * w); };

    // the host's clock: the time record may already be the launch's last
    // (written by CTA 0) when a CTA far from it starts
    double T = r.T0, Tbefore = T;
    const bool exported = i_own < nm && __ldg(r.exported + g_own) != 0;
    // FP32 forms: the first halo masses of the first pass (the loads of their
    // records then wait for nothing else)
    constexpr int kAhead = PREC == P_FP64 ? 0 : 2;
    int32_t hx[kAhead + 1];
#pragma unroll
    for (int k = 0; k < kAhead; k++) {
        const int v = threadIdx.x + k * blockDim.x;
        hx[k] = v < nh * kVec ? __ldg(a.halo + ti.halo_off + v / kVec) : 0;
    }

    if (single) grid_dep_wait();
    if constexpr (PREC != P_FP64) load_tile();
    St<PREC> rk0;  // RK2: the step's starting state
    if (PREC != P_FP64 && INTEG == INTEG_RK2 && r.half && i_own < nm)  // in the buffer this launch writes
        rk0 = load_state<PREC, true>(parity ? a.state0 : a.state1, g_own);
    R acc0[3] = {0, 0, 0};  // VERLET: the acceleration of the step before
    if (INTEG == INTEG_VERLET && !(fl & MF_FIXED)) {
#pragma unroll
        for (int c = 0; c < 3; c++) acc0[c] = PREC == P_FP64 ? reinterpret_cast<const R *>(a.acc)[c * np + g_own]
                                     : load_fresh<PREC>(reinterpret_cast<const R *>(a.acc) + c * np + g_own);
    }
    LaneMass lm{};
    double lx = 0.0, lv = 0.0;  // the lane's position and velocity
    if constexpr (LANES) {
        lm.c = c_sp;
        lm.j = lane % kLaneMasses;
        lm.g = (int64_t)ti.mass_off + i_sp;
        lm.m = 1.0;
        if (i_sp < nm) {
            lm.fl = __ldg(a.flags + lm.g);
            lm.on = !(lm.fl & MF_FIXED);
            lm.m = (double)__ldg(reinterpret_cast<const R *>(a.mass) + lm.g);
            const double *q = reinterpret_cast<const double *>(parity ? a.state1 : a.state0) + 6 * lm.g;
            lx = q[c_sp];
            lv = q[3 + c_sp];
            if (INTEG == INTEG_VERLET) lm.acc0 = reinterpret_cast<const double *>(a.acc)[c_sp * np + lm.g];
        }
        lm.gm = a.prm->g[c_sp] * lm.m;
        uint32_t bad = 0;
        const Alu y = alu_unpack(lm.m, bad);
        lm.md = alu_divisor(y);
        lm.md_ok = !alu_bad(bad) && alu_nonzero(y);
    }
    const bool lane_exported = LANES && lm.on && __ldg(r.exported + lm.g) != 0;
    for (int64_t pass = 0; pass < passes; pass++) {
        // ---- A: the halo's records of the pass before ------------------------
        bool gave_up = false;
        if (pass > 0) {
            const uint8_t *xin = r.xbuf + (int64_t)(pass & 1) * r.xbytes;
            const uint32_t tag = r.base + (uint32_t)pass;
            const int nq = nh * kChunks;
            for (int q0 = threadIdx.x; q0 < nq && !gave_up; q0 += kPoll * blockDim.x) {
                const uint8_t *src[kPoll];
                uint32_t todo = 0;
#pragma unroll
                for (int k = 0; k < kPoll; k++) {
                    const int q = q0 + k * blockDim.x;
                    const int32_t g = q < nq ? __ldg(r.halo + ti.halo_off + q / kChunks) : -1;  // -1: fixed
                    src[k] = xin + ((int64_t)g * kChunks + q % kChunks) * 16;
                    if (g >= 0) todo |= 1u << k;
                }
                for (uint32_t it = 0; todo; it++) {
                    Chunk x[kPoll];
#pragma unroll
                    for (int k = 0; k < kPoll; k++)
                        if (todo >> k & 1) x[k] = ld_chunk(src[k]);
#pragma unroll
                    for (int k = 0; k < kPoll; k++)
                        if ((todo >> k & 1) && x[k].tag == tag) {
                            const int q = q0 + k * blockDim.x;
                            uint32_t *dst = reinterpret_cast<uint32_t *>(st + (int64_t)(nm + q / kChunks) * kRec) +
                                            3 * (q % kChunks);
                            dst[0] = x[k].w[0];
                            dst[1] = x[k].w[1];
                            dst[2] = x[k].w[2];
                            todo &= ~(1u << k);
                        }
                    if (it == r.last_poll ||
                        ((it & 1023u) == 1023u && *reinterpret_cast<const volatile int *>(a.err))) {
                        gave_up = todo != 0;
                        break;
                    }
                }
            }
        } else {
            const uint8_t *in = reinterpret_cast<const uint8_t *>(parity ? a.state1 : a.state0);
            float4 *const to = reinterpret_cast<float4 *>(st + (int64_t)nm * kRec);
            auto rec = [&](int32_t h, int v) {
                return load_fresh<PREC>(reinterpret_cast<const float4 *>(in + (int64_t)h * kRec) + v % kVec);
            };
            int v = threadIdx.x;
#pragma unroll
            for (int k = 0; k < kAhead; k++, v += blockDim.x)
                if (v < nh * kVec) to[v] = rec(hx[k], v);
            for (; v < nh * kVec; v += blockDim.x) to[v] = rec(__ldg(a.halo + ti.halo_off + v / kVec), v);
        }
        if (__syncthreads_or(gave_up)) {
            if (threadIdx.x == 0) atomicOr(a.err, 1);
            return;
        }

        // ---- B: one force per slab entry --------------------------------
        const StepTime tm = step_time(T);
        for (int e0 = threadIdx.x; e0 < E; e0 += kBatch * blockDim.x) {
            Rec16<PREC> rc[kBatch], q[kBatch];
#pragma unroll
            for (int k = 0; k < kBatch; k++) {
                const int e = e0 + k * blockDim.x;
                if (e < E)
                    rc[k] = STAGE ? load_rec<PREC>(smem + L.ent + (int64_t)e * kSlot)
                                  : ldg_rec<PREC>(gent + (int64_t)e * kSlot);
                if (e < ti.nact)
                    q[k] = STAGE ? load_rec<PREC>(smem + L.act + (int64_t)e * kSlot)
                                 : ldg_rec<PREC>(gact + (int64_t)e * kSlot);
            }
#pragma unroll
            for (int k = 0; k < kBatch; k++) {
                const int e = e0 + k * blockDim.x;
                if (e < E) entry_force<PREC>(rc[k], e < ti.nact, q[k], st, tm, slots + (int64_t)e * kSlot);
            }
        }
        __syncthreads();

        // ---- C: sums, constraints, integration --------------------------
        if (ti.nheavy > 0) {
            heavy_sums<PREC>(a, ti, slots, sH, threadIdx.x >> 5, blockDim.x >> 5);
            __syncthreads();
        }
        if constexpr (LANES) {
            if (warp * kLaneMasses < nm) {
                double F = 0;
                if (d_sp == 255) {
                    int h = 0;
                    while (h < ti.nheavy && a.heavy_local[ti.heavy_off + h] != i_sp) h++;
                    F = F + (double)sH[c_sp * ti.nheavy + h];
                } else if (i_sp < nm) {
                    F = gather_list_component(slots, nw, word, c_sp);
                }
                __syncwarp();
                integrate_lanes<INTEG>(a, ti, prm, lm, F, lx, lv, write_acc && pass == passes - 1,
                                       INTEG == INTEG_RK2 ? (int)(pass & 1) : 0);
                if (lm.on) {
                    double *q = reinterpret_cast<double *>(st + (int64_t)i_sp * kRec);
                    q[c_sp] = lx;
                    q[3 + c_sp] = lv;
                    if (pass == passes - 1) {
                        double *o = reinterpret_cast<double *>((parity ^ (int)(passes & 1)) ? a.state1 : a.state0) + 6 * lm.g;
                        o[c_sp] = lx;
                        o[3 + c_sp] = lv;
                    }
                }
                __syncwarp();
                if (pass < passes - 1) {
                    // the warp's records to the exchange, a chunk per lane
                    const uint32_t tag = r.base + (uint32_t)pass + 1;
                    const uint32_t ex = __ballot_sync(0xffffffffu, lane_exported);
                    for (int q = lane; q < kLaneMasses * kChunks; q += 32) {
                        const int k = q / kChunks, c = q % kChunks, i = warp * kLaneMasses + k;
                        if (!(ex >> k & 1)) continue;  // lane k has mass k's first component
                        const uint32_t *w = reinterpret_cast<const uint32_t *>(st + (int64_t)i * kRec) + 3 * c;
                        st_chunk(r.xbuf + (int64_t)((pass + 1) & 1) * r.xbytes +
                                     (((int64_t)ti.mass_off + i) * kChunks + c) * 16,
                                 Chunk{{w[0], w[1], w[2]}, tag});
                    }
                }
            }
            Tbefore = T;
            T = T + prm->launch_dt;
            continue;
        }
        if (split) {
            if (i_sp < nm) sF[c_sp * nm + i_sp] = gather_list_component(slots, nw, word, c_sp);
            __syncthreads();
        }
        if (!(fl & MF_FIXED)) {  // src/sim.cu:1100
            R F0 = 0, F1 = 0, F2 = 0;
            if (d == 255) {
                int h = 0;
                while (h < ti.nheavy && a.heavy_local[ti.heavy_off + h] != i_own) h++;
                F0 = F0 + sH[h];
                F1 = F1 + sH[ti.nheavy + h];
                F2 = F2 + sH[2 * ti.nheavy + h];
            } else if (split) {
                F0 = (R)sF[i_own];
                F1 = (R)sF[nm + i_own];
                F2 = (R)sF[2 * nm + i_own];
            } else {
                for (uint32_t w = 0; w < nw; w++) gather_word_padded<PREC>(slots, word(w), F0, F1, F2);
            }
            St<PREC> s = load_state_smem<PREC>(st, i_own);
            const int rk2_stage = INTEG == INTEG_RK2 ? (int)(pass & 1) ^ (PREC == P_FP64 ? 0 : r.half) : 0;
            if (INTEG == INTEG_RK2 && rk2_stage == 0) rk0 = s;
            integrate<PREC, INTEG>(a, ti, g_own, fl, m, F0, F1, F2, s, st, i_own, write_acc && pass == passes - 1, np,
                                   prm, rk2_stage, &rk0, INTEG == INTEG_VERLET ? acc0 : nullptr);
            if (exported && pass < passes - 1) {
                uint32_t w[12];
                record_words<PREC>(s, w);
                uint8_t *x = r.xbuf + (int64_t)((pass + 1) & 1) * r.xbytes + g_own * (kChunks * 16);
                const uint32_t tag = r.base + (uint32_t)pass + 1;
#pragma unroll
                for (int c = 0; c < kChunks; c++) st_chunk(x + 16 * c, Chunk{{w[3 * c], w[3 * c + 1], w[3 * c + 2]}, tag});
            }
            if (pass == passes - 1)
                store_state<PREC>((parity ^ (int)(passes & 1)) ? a.state1 : a.state0, g_own, s);
        }
        Tbefore = T;
        T = T + prm->launch_dt;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        const int p = parity ^ (int)(passes & 1);
        a.tbuf[p] = T;
        a.tbuf[p ^ 1] = Tbefore;
    }
}

template <int PREC, int INTEG, bool LANES>
const void *rg_kernel(int stage, int shape) {
    static const void *const f[2][kGridShapes] = {
        {(const void *)k_grid_resident<PREC, INTEG, 0, 0, LANES>, (const void *)k_grid_resident<PREC, INTEG, 0, 1, LANES>,
         (const void *)k_grid_resident<PREC, INTEG, 0, 2, LANES>},
        {(const void *)k_grid_resident<PREC, INTEG, 1, 0, LANES>, (const void *)k_grid_resident<PREC, INTEG, 1, 1, LANES>,
         (const void *)k_grid_resident<PREC, INTEG, 1, 2, LANES>}};
    return f[stage][shape];
}
// the kernel of an integrator, staging and launch shape
template <int PREC, bool LANES>
const void *rg_kernel(int integ, int stage, int shape) {
    switch (integ) {
        case INTEG_VERLET: return rg_kernel<PREC, INTEG_VERLET, LANES>(stage, shape);
        case INTEG_RK2: return rg_kernel<PREC, INTEG_RK2, LANES>(stage, shape);
        default: return rg_kernel<PREC, INTEG_EULER, LANES>(stage, shape);
    }
}
}  // namespace
}  // namespace tg
