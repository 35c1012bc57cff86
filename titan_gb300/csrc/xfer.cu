// xfer.cu -- per-mass transfer between caller order and tiled order
// (get/set/getAll/setAll: src/sim.cu:588-764 in the reference) and the FP64
// energy / momentum diagnostics (test/testutil/utils.h:12-43).
#include <cstdint>

#include "engine.h"
#include "state.cuh"
#include "step_math.cuh"

namespace tg {

namespace {

// ------------------------------------------------- gather / scatter -------
// The outputs may be page-locked host memory: a warp exchanges its 32 masses'
// triples by shuffles and writes them as consecutive doubles, so that a read
// of a small scene is this one kernel (a copy per array and one for the error
// flag took 55 us a call, this 25) and a large one moves at the link's rate
// while it gathers.  No shared memory and few registers: the request loop
// (server.cu) leaves 6,688 bytes and a quarter of the register file on each
// SM, and reads of finished scenes have to run beside it.
constexpr int kGatherBlock = 256;
__device__ __forceinline__ void store_triples(double *out, int64_t i0, int64_t count, double x0, double x1, double x2) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int r = 0; r < 3; r++) {
        const int e = 32 * r + lane, src = e / 3, c = e - 3 * src;
        const double y0 = __shfl_sync(0xffffffffu, x0, src), y1 = __shfl_sync(0xffffffffu, x1, src),
                     y2 = __shfl_sync(0xffffffffu, x2, src);
        if (i0 + src < count) out[3 * i0 + e] = c == 0 ? y0 : (c == 1 ? y1 : y2);
    }
}
template <int PREC>
__global__ void __launch_bounds__(kGatherBlock) k_gather(XferArgs a) {
    using R = typename Real<PREC>::T;
    const int64_t i = (int64_t)blockIdx.x * kGatherBlock + threadIdx.x, i0 = i - (threadIdx.x & 31);
    if (i == 0 && a.err_out) *a.err_out = *a.err;
    if (i0 >= a.count) return;  // whole warps
    // lanes past the end repeat the last mass and store nothing
    const int64_t j = i < a.count ? i : a.count - 1;
    const int64_t g = a.old2new[a.idx ? a.idx[j] : j];
    if (a.pos || a.vel) {
        const St<PREC> s = load_state<PREC>(a.parity ? a.state1 : a.state0, g);
        double x[3], v[3];
#pragma unroll
        for (int c = 0; c < 3; c++) {
            x[c] = (double)s.x[c], v[c] = (double)s.v[c];
            if constexpr (PREC == P_FP32C) {
                x[c] += (double)s.xl[c];
                v[c] += (double)s.vl[c];
            }
        }
        if (a.pos) store_triples(a.pos, i0, a.count, x[0], x[1], x[2]);
        if (a.vel) store_triples(a.vel, i0, a.count, v[0], v[1], v[2]);
    }
    if (a.accout) {
        const R *acc = reinterpret_cast<const R *>(a.acc) + g;
        store_triples(a.accout, i0, a.count, (double)acc[0], (double)acc[a.npad], (double)acc[2 * a.npad]);
    }
}

// Positions of all masses in caller (creation) order as float triples, the
// headless form of the reference's updateVertices (src/sim.cu:1717-1725):
// (float) of the position (FP32C: of hi + lo in double).
template <int PREC>
__global__ void k_export_f32(XferArgs a, float *out) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.count) return;
    const int64_t g = a.old2new[i];
    const St<PREC> s = load_state<PREC>(a.parity ? a.state1 : a.state0, g);
#pragma unroll
    for (int c = 0; c < 3; c++) {
        double x = (double)s.x[c];
        if constexpr (PREC == P_FP32C) x += (double)s.xl[c];
        out[3 * i + c] = (float)x;
    }
}

// Writes pos and/or vel of the listed masses into both buffers, keeping the
// other field from the current buffer.
template <int PREC>
__global__ void k_scatter(XferArgs a) {
    using R = typename Real<PREC>::T;
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.count) return;
    int64_t src = a.idx ? a.idx[i] : i;
    int64_t g = a.old2new[src];
    const int64_t np = a.npad;
    St<PREC> s = load_state<PREC>(a.parity ? a.state1 : a.state0, g);
#pragma unroll
    for (int c = 0; c < 3; c++) {
        if (a.ipos) {
            double x = a.ipos[3 * i + c];
            s.x[c] = (R)x;
            if constexpr (PREC == P_FP32C) s.xl[c] = (R)(x - (double)s.x[c]);
        }
        if (a.ivel) {
            double v = a.ivel[3 * i + c];
            s.v[c] = (R)v;
            if constexpr (PREC == P_FP32C) s.vl[c] = (R)(v - (double)s.v[c]);
        }
        if (a.ipos) reinterpret_cast<R *>(a.acc)[c * np + g] = (R)0;
    }
    store_state<PREC>(a.state0, g, s);
    store_state<PREC>(a.state1, g, s);
}

// Raw state records and accelerations to (out) or from caller order, bit for
// bit: a plan's state carried over to another plan of the same masses.
template <bool OUT>
__global__ void __launch_bounds__(256) k_carry(XferArgs a, float4 *rec, uint32_t *acc, int vecs, int words) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.count) return;
    const int64_t g = a.old2new[i];
    float4 *const s0 = reinterpret_cast<float4 *>(a.state0) + g * vecs, *const s1 = reinterpret_cast<float4 *>(a.state1) + g * vecs;
    for (int v = 0; v < vecs; v++) {
        if (OUT) rec[i * vecs + v] = (a.parity ? s1 : s0)[v];
        else s0[v] = s1[v] = rec[i * vecs + v];
    }
    for (int c = 0; c < 3; c++)
        for (int w = 0; w < words; w++) {
            uint32_t *const x = reinterpret_cast<uint32_t *>(a.acc) + (c * a.npad + g) * words + w;
            uint32_t *const y = acc + (c * a.count + i) * words + w;
            if (OUT) *y = *x;
            else *x = *y;
        }
}

// ------------------------------------------------- entry records ----------
// One thread per slab entry: the fields of its record and actuation record
// whose parameters are given, with the host's conversions (upload_records in
// capi.cu).  Bound by the gathers of 8-byte parameters (a tile's entries are
// near in creation order) and the strided stores.
template <int PREC>
__global__ void __launch_bounds__(256) k_entries(EntryArgs a) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= a.count) return;
    const int32_t j = a.spring[e];
    if (j < 0) return;
    if constexpr (PREC == P_FP64) {
        double *rec = reinterpret_cast<double *>(a.rec) + 4 * e, *act = reinterpret_cast<double *>(a.act) + 4 * e;
#pragma unroll
        for (int q = 0; q < 3; q++) {
            if (a.par[q]) rec[q] = a.par[q][j];
            if (a.par[3 + q]) act[q] = a.par[3 + q][j];
        }
    } else {
        float *rec = reinterpret_cast<float *>(a.rec) + 4 * e, *act = reinterpret_cast<float *>(a.act) + 4 * e;
        constexpr double kTwoPi = 6.283185307179586476925286766559;
#pragma unroll
        for (int q = 0; q < 3; q++)
            if (a.par[q]) rec[1 + q] = (float)a.par[q][j];
        if (a.par[1]) act[3] = (float)a.par[1][j];
        if (a.par[3]) act[0] = (float)(a.par[3][j] / kTwoPi);
        if (a.par[4]) {
            const uint32_t type = __float_as_uint(rec[0]) >> 24 & 3u;
            act[1] = (float)(type == 2 ? -a.par[4][j] : a.par[4][j]);
        }
        if (a.par[5]) act[2] = (float)(a.par[5][j] / kTwoPi);
    }
}

// One thread per repeated entry: its source's record and actuation record, the
// entry word's type bits with the ends given.
template <int PREC>
__global__ void __launch_bounds__(256) k_repeat_entries(RepeatArgs a) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= a.count) return;
    constexpr int kVec = PREC == P_FP64 ? 2 : 1;
    float4 *const rec = reinterpret_cast<float4 *>(a.rec), *const act = reinterpret_cast<float4 *>(a.act);
    const int64_t from = (int64_t)a.src[e] * kVec, to = (a.first + e) * kVec;
#pragma unroll
    for (int v = 0; v < kVec; v++) {
        float4 r = rec[from + v];
        // the entry word: FP64 the low half of the last double, FP32 the first float
        float &w = PREC == P_FP64 ? r.z : r.x;
        if (v == kVec - 1)
            w = __uint_as_float((__float_as_uint(w) & 0xff000000u) | (a.ends[e] & 0x00ffffffu));
        rec[to + v] = r;
        act[to + v] = act[from + v];
    }
}

// ------------------------------------------------------ diagnostics -------
// Pass 1: each of kDiagBlocks blocks sums a fixed grid-stride share in FP64
// and reduces it with a fixed tree; pass 2 reduces the partials the same way.
// The lengths' products and square roots are on the integer units
// (fp64_alu.cuh).
template <int PREC>
__global__ void __launch_bounds__(256) k_diag1(DiagArgs a) {
    __shared__ double red[kDiagQ][256];
    double q[kDiagQ];
#pragma unroll
    for (int k = 0; k < kDiagQ; k++) q[k] = 0.0;
    using R = typename Real<PREC>::T;
    const R *ms = reinterpret_cast<const R *>(a.mass);
    auto pos = [&](const St<PREC> &s, int c) {
        double x = (double)s.x[c];
        if constexpr (PREC == P_FP32C) x += (double)s.xl[c];
        return x;
    };
    auto vel = [&](const St<PREC> &s, int c) {
        double v = (double)s.v[c];
        if constexpr (PREC == P_FP32C) v += (double)s.vl[c];
        return v;
    };
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g < a.n; g += stride) {
        const St<PREC> s = load_state<PREC>(a.state, g);
        double m = (double)ms[g];
        double x[3] = {pos(s, 0), pos(s, 1), pos(s, 2)};
        double v[3] = {vel(s, 0), vel(s, 1), vel(s, 2)};
        double vn = nrm3_alu(v[0], v[1], v[2]);
        q[1] += (0.5 * m) * (vn * vn);
        q[2] += (a.g_mag * x[2]) * m;
        double p[3] = {v[0] * m, v[1] * m, v[2] * m};
        q[3] += p[0];
        q[4] += p[1];
        q[5] += p[2];
        q[6] += p[1] * x[2] - p[2] * x[1];
        q[7] += x[0] * p[2] - p[0] * x[2];
        q[8] += p[0] * x[1] - p[1] * x[0];
    }
    for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < a.ns; s += stride) {
        int32_t l = a.sl[s], r = a.sr[s];
        if (l < 0) continue;
        const St<PREC> sl = load_state<PREC>(a.state, l), sr = load_state<PREC>(a.state, r);
        double d0 = pos(sl, 0) - pos(sr, 0), d1 = pos(sl, 1) - pos(sr, 1), d2 = pos(sl, 2) - pos(sr, 2);
        double x = nrm3_alu(d0, d1, d2) - a.srest[s];
        q[0] += (a.sk[s] * (x * x)) / 2;
    }
#pragma unroll
    for (int k = 0; k < kDiagQ; k++) red[k][threadIdx.x] = q[k];
    __syncthreads();
    for (int w = 128; w >= 1; w >>= 1) {
        if ((int)threadIdx.x < w)
            for (int k = 0; k < kDiagQ; k++) red[k][threadIdx.x] += red[k][threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x < kDiagQ) a.partials[blockIdx.x * kDiagQ + threadIdx.x] = red[threadIdx.x][0];
}

__global__ void __launch_bounds__(256) k_diag2(DiagArgs a) {
    __shared__ double red[kDiagQ][256];
    for (int k = 0; k < kDiagQ; k++) {
        double s = 0.0;
        for (int b = threadIdx.x; b < kDiagBlocks; b += 256) s += a.partials[b * kDiagQ + k];
        red[k][threadIdx.x] = s;
    }
    __syncthreads();
    for (int w = 128; w >= 1; w >>= 1) {
        if ((int)threadIdx.x < w)
            for (int k = 0; k < kDiagQ; k++) red[k][threadIdx.x] += red[k][threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x < kDiagQ) a.out[threadIdx.x] = red[threadIdx.x][0];
}

}  // namespace


template <int PREC>
static cudaError_t load_transfers() {
    const void *const f[] = {(const void *)k_gather<PREC>, (const void *)k_scatter<PREC>,
                             (const void *)k_export_f32<PREC>, (const void *)k_entries<PREC>};
    cudaError_t e = cudaSuccess;
    cudaFuncAttributes at;
    for (const void *k : f)
        if (e == cudaSuccess) e = cudaFuncGetAttributes(&at, k);
    return e;
}
// A kernel's first use loads its code, and that waits for running kernels --
// beside the request loop, until the loop leaves.
cudaError_t xfer_prepare(int precision) {
    return precision == P_FP64   ? load_transfers<P_FP64>()
           : precision == P_FP32 ? load_transfers<P_FP32>()
                                 : load_transfers<P_FP32C>();
}

cudaError_t launch_export_f32(int precision, const XferArgs &a, float *out, cudaStream_t s) {
    if (a.count <= 0) return cudaSuccess;
    const unsigned blocks = (unsigned)((a.count + 255) / 256);
    switch (precision) {
        case P_FP64: k_export_f32<P_FP64><<<blocks, 256, 0, s>>>(a, out); break;
        case P_FP32: k_export_f32<P_FP32><<<blocks, 256, 0, s>>>(a, out); break;
        default: k_export_f32<P_FP32C><<<blocks, 256, 0, s>>>(a, out); break;
    }
    return cudaGetLastError();
}

cudaError_t launch_gather(int precision, const XferArgs &a, cudaStream_t s) {
    if (a.count <= 0) return cudaSuccess;
    const int blocks = (int)((a.count + kGatherBlock - 1) / kGatherBlock);
    switch (precision) {
        case P_FP64: k_gather<P_FP64><<<blocks, kGatherBlock, 0, s>>>(a); break;
        case P_FP32: k_gather<P_FP32><<<blocks, kGatherBlock, 0, s>>>(a); break;
        default: k_gather<P_FP32C><<<blocks, kGatherBlock, 0, s>>>(a); break;
    }
    return cudaGetLastError();
}

cudaError_t launch_scatter(int precision, const XferArgs &a, cudaStream_t s) {
    if (a.count <= 0) return cudaSuccess;
    int blocks = (int)((a.count + 255) / 256);
    switch (precision) {
        case P_FP64: k_scatter<P_FP64><<<blocks, 256, 0, s>>>(a); break;
        case P_FP32: k_scatter<P_FP32><<<blocks, 256, 0, s>>>(a); break;
        default: k_scatter<P_FP32C><<<blocks, 256, 0, s>>>(a); break;
    }
    return cudaGetLastError();
}

cudaError_t launch_carry(int precision, const XferArgs &a, bool out, void *rec, void *acc, cudaStream_t s) {
    if (a.count <= 0) return cudaSuccess;
    const unsigned blocks = (unsigned)((a.count + 255) / 256);
    const int vecs = state_record_bytes(precision) / 16, words = precision == P_FP64 ? 2 : 1;
    if (out) k_carry<true><<<blocks, 256, 0, s>>>(a, (float4 *)rec, (uint32_t *)acc, vecs, words);
    else k_carry<false><<<blocks, 256, 0, s>>>(a, (float4 *)rec, (uint32_t *)acc, vecs, words);
    return cudaGetLastError();
}

cudaError_t launch_entries(int precision, const EntryArgs &a, cudaStream_t s) {
    if (a.count <= 0) return cudaSuccess;
    const unsigned blocks = (unsigned)((a.count + 255) / 256);
    switch (precision) {
        case P_FP64: k_entries<P_FP64><<<blocks, 256, 0, s>>>(a); break;
        case P_FP32: k_entries<P_FP32><<<blocks, 256, 0, s>>>(a); break;
        default: k_entries<P_FP32C><<<blocks, 256, 0, s>>>(a); break;
    }
    return cudaGetLastError();
}

cudaError_t launch_repeat_entries(int precision, const RepeatArgs &a, cudaStream_t s) {
    if (a.count <= 0) return cudaSuccess;
    const unsigned blocks = (unsigned)((a.count + 255) / 256);
    switch (precision) {
        case P_FP64: k_repeat_entries<P_FP64><<<blocks, 256, 0, s>>>(a); break;
        case P_FP32: k_repeat_entries<P_FP32><<<blocks, 256, 0, s>>>(a); break;
        default: k_repeat_entries<P_FP32C><<<blocks, 256, 0, s>>>(a); break;
    }
    return cudaGetLastError();
}

cudaError_t launch_diag(int precision, const DiagArgs &a, cudaStream_t s) {
    switch (precision) {
        case P_FP64: k_diag1<P_FP64><<<kDiagBlocks, 256, 0, s>>>(a); break;
        case P_FP32: k_diag1<P_FP32><<<kDiagBlocks, 256, 0, s>>>(a); break;
        default: k_diag1<P_FP32C><<<kDiagBlocks, 256, 0, s>>>(a); break;
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    k_diag2<<<1, 256, 0, s>>>(a);
    return cudaGetLastError();
}

}  // namespace tg
