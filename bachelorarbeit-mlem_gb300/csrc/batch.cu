// batch.cu — many sinograms against one resident matrix (batched SpMM).
//
// The matrix stream is shared by the instances of a tile (BT = 8, 16 or 32
// slots, interleaved: slot b of voxel c is f[c*BT + b]).  A launch covers the
// first W slots (the active width, 4..BT, the smallest power of two holding
// every slot with iterations left): a row is handled by a segment of W lanes
// of a warp (32/W rows per warp); each lane owns 4 instances of a nonzero and
// reads their image entries with one 16-byte load, so W/4 lanes cover a
// nonzero and a segment takes 4 nonzeros per gather instruction.
//
// Every instance sums its row in 4 chains: the row's 4-entry vectors (aligned
// to multiples of 4 entries of the matrix) go to the chains in turn, each chain
// a sequential FMA chain in entry order, combined as (c0 + c1) + (c2 + c3).  The
// W/4 lanes of a chain load its vectors of indices and values themselves (one
// request each per instruction).  That order depends on neither W nor BT nor
// the slot, so an instance gives the same bits alone and in a full batch, in
// any tile.
//
// What bounds it: the latency of a nonzero's gather of the slots' state, one
// 128-byte line with 32 slots, mostly from L2 (28% L1 hits in the forward, 68% in
// the back projection), at the 67-71% of the warps that 40 registers leave; no
// unit is saturated (L1 data pipe 65-67%, issue 35%).  Handing 32 coalesced entries
// round with shuffles, as an earlier form did, put 2 shuffles on the L1 data pipe
// for every 4 nonzeros: one iteration of the 3-D mid matrix with 4 / 8 / 16 / 32
// slots 1.28 / 1.38 / 2.01 / 3.25 -> 1.19 / 1.35 / 1.88 / 3.12 ms (FP16 values 1.28 /
// 1.36 / 1.97 / 3.22 -> 1.14 / 1.30 / 1.87 / 2.98), of a matrix of 6 M nonzeros 0.134 /
// 0.136 / 0.200 / 0.310 -> 0.131 / 0.136 / 0.181 / 0.278 ms; 24 sinograms of 5 to 20
// iterations on the mid matrix 54.5 -> 51.4 ms.  6 blocks per SM (40
// registers), one vector at a time; measured and not kept, 16 / 32 slots on the
// mid matrix: 8 blocks (32 registers, spills) 2.41 / 3.76, 5 blocks 1.94 / 3.25,
// the next vector loaded before the gathers 2.24 / 3.83 (5 blocks 1.99 / 3.31),
// two vectors unrolled with 5 and 4 blocks 1.95 / 3.28 and 2.02 / 3.38 ms.
//
// Per-slot iteration counters live on the device (remaining[b]); an
// iteration is FP, BP+update and a counter tick, replayable as one CUDA
// graph per width; a slot whose counter reached 0 is no longer updated.
#include "kernels.cuh"

#include <algorithm>

namespace mlem {

namespace {

// Row sums of one warp's 32/W rows (segment seg of W lanes holds row `row`,
// `ok` = the row exists).  On return the lanes sl < W/4 of each segment hold
// instances 4*sl..4*sl+3 of their row.
// NC: the gathered state is read through the read-only path (__ldg), which is
// right only when no block of the same launch writes it; the persistent loop
// below, whose phases write what the next phase gathers, uses plain loads.
template <bool NC>
__device__ __forceinline__ float4 load_state(const char* p) {
    if (NC) return __ldg(reinterpret_cast<const float4*>(p));
    return *reinterpret_cast<const float4*>(p);
}

__device__ __forceinline__ void fma_state(float4& acc, float v, const float4& x) {
    acc.x = fmaf(v, x.x, acc.x);
    acc.y = fmaf(v, x.y, acc.y);
    acc.z = fmaf(v, x.z, acc.z);
    acc.w = fmaf(v, x.w, acc.w);
}

template <typename V, int W, bool NC = true>
__device__ __forceinline__ void batch_rows(const uint64_t* __restrict__ rowptr, const uint32_t* __restrict__ idx,
                                           const V* __restrict__ val, const float* x, uint32_t BT, uint32_t na,
                                           uint32_t row, bool ok, int lane, float4& acc) {
    constexpr int LPN = W / 4;  // lanes per nonzero
    const int sl = lane % W, chain = sl / LPN;
    const uint32_t q4 = (sl % LPN) * 4;
    // lanes of slots that are not read repeat those of slot 0 (no bytes of their own)
    const char* xq = reinterpret_cast<const char*>(x + (q4 < na ? q4 : 0));
    const uint32_t stride = BT * (uint32_t)sizeof(float);
    uint64_t s = 0, t = 0;
    if (ok) {
        s = rowptr[row];
        t = rowptr[row + 1];
    }
    if (s < t) {
        const uint64_t v0 = s >> 2;
        const uint4* ip = reinterpret_cast<const uint4*>(idx) + v0;
        const V* vp = val + 4 * v0;
        const uint32_t lo = (uint32_t)(s & 3), hi = (uint32_t)(t - 4 * v0);  // the row's entries, relative to 4 v0
        auto part = [&](uint32_t v) {  // a vector that is not all the row's
            const uint4 c = ld_stream(ip + v);
            float a[4];
            Val4<V>::load(vp, v, a);
            const uint32_t cs[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (4 * v + k >= lo && 4 * v + k < hi)
                    fma_state(acc, a[k], load_state<NC>(xq + (uint64_t)cs[k] * stride));
        };
        const uint32_t whole = hi >> 2;
        uint32_t v = chain;
        if (v == 0 && lo) {
            part(0);
            v = 4;
        }
#pragma unroll 1
        for (; v < whole; v += 4) {
            const uint4 c = ld_stream(ip + v);
            float a[4];
            Val4<V>::load(vp, v, a);
            const uint32_t cs[4] = {c.x, c.y, c.z, c.w};
            float4 xv[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) xv[k] = load_state<NC>(xq + (uint64_t)cs[k] * stride);
#pragma unroll
            for (int k = 0; k < 4; ++k) fma_state(acc, a[k], xv[k]);
        }
        if (v == whole && (hi & 3)) part(v);
    }
    __syncwarp();
    // (c0 + c1) + (c2 + c3): chains sit LPN lanes apart inside the segment
#pragma unroll
    for (int o = LPN; o < W; o <<= 1) {
        acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
        acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
        acc.z += __shfl_xor_sync(0xffffffffu, acc.z, o);
        acc.w += __shfl_xor_sync(0xffffffffu, acc.w, o);
    }
}

__device__ __forceinline__ float correl1(int32_t g, float fp) { return (fp != 0.0f) ? __fdiv_rn((float)g, fp) : 0.0f; }

__device__ __forceinline__ float update1(float f, float acc, float n) {
    const float t = __fmul_rn(f, acc);
    return (n == 0.0f) ? t : __fdiv_rn(t, n);
}

// ratio[row*BT + b] = g/(A f)_b for the first W slots.
template <typename V, int W>
__global__ void __launch_bounds__(256, 6)
k_batch_fp(const uint64_t* __restrict__ rowptr, const uint32_t* __restrict__ idx,
           const V* __restrict__ val, const float* __restrict__ f, uint32_t rows, uint32_t BT, uint32_t na,
           const int32_t* __restrict__ g, float* __restrict__ ratio) {
    const int lane = threadIdx.x & 31;
    const uint64_t first = ((blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5) * (32 / W);
    if (first >= rows) return;  // whole warp
    const uint64_t row = first + lane / W;
    const bool ok = row < rows;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    batch_rows<V, W>(rowptr, idx, val, f, BT, na, (uint32_t)row, ok, lane, acc);
    const int sl = lane % W;
    if (ok && sl < W / 4 && (uint32_t)sl * 4 < na) {
        const uint64_t o = row * BT + sl * 4;
        const int4 gg = *reinterpret_cast<const int4*>(g + o);
        *reinterpret_cast<float4*>(ratio + o) =
            make_float4(correl1(gg.x, acc.x), correl1(gg.y, acc.y), correl1(gg.z, acc.z), correl1(gg.w, acc.w));
    }
}

// f[c*BT + b] = f·(Aᵀ ratio)_b / norm[c] for the slots b < W with iterations left.
template <typename V, int W>
__global__ void __launch_bounds__(256, 6)
k_batch_bp(const uint64_t* __restrict__ rowptr, const uint32_t* __restrict__ idx,
           const V* __restrict__ val, const float* __restrict__ ratio, uint32_t cols, uint32_t BT, uint32_t na,
           const float* __restrict__ norm, const uint32_t* __restrict__ remaining,
           float* __restrict__ f) {
    const int lane = threadIdx.x & 31;
    const uint64_t first = ((blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5) * (32 / W);
    if (first >= cols) return;  // whole warp
    const uint64_t c = first + lane / W;
    const bool ok = c < cols;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    batch_rows<V, W>(rowptr, idx, val, ratio, BT, na, (uint32_t)c, ok, lane, acc);
    const int sl = lane % W;
    if (ok && sl < W / 4 && (uint32_t)sl * 4 < na) {
        const uint64_t o = c * BT + sl * 4;
        const uint4 rem = *reinterpret_cast<const uint4*>(remaining + sl * 4);
        const float n = norm[c];
        float4 fv = *reinterpret_cast<const float4*>(f + o);
        if (rem.x) fv.x = update1(fv.x, acc.x, n);
        if (rem.y) fv.y = update1(fv.y, acc.y, n);
        if (rem.z) fv.z = update1(fv.z, acc.z, n);
        if (rem.w) fv.w = update1(fv.w, acc.w, n);
        *reinterpret_cast<float4*>(f + o) = fv;
    }
}

template <typename V, int BT>
__global__ void __launch_bounds__(256)
k_batch_scatter(const uint64_t* __restrict__ rowptr, const uint32_t* __restrict__ idx,
                const V* __restrict__ val, const float* __restrict__ ratio, uint32_t rows,
                float* __restrict__ bp) {
    constexpr int G = 32 / BT;
    const uint32_t row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31, grp = lane / BT, b = lane % BT;
    if (row >= rows) return;
    const float r = ratio[(uint64_t)row * BT + b];
    const uint64_t s = rowptr[row], t = rowptr[row + 1];
    for (uint64_t base = s; base < t; base += 32) {
        const uint64_t e = base + lane;
        uint32_t c = 0;
        float v = 0.f;
        if (e < t) {
            c = ld_stream(idx + e);
            v = Val4<V>::one(val, e);
        }
        const int n = (t - base) > 32 ? 32 : (int)(t - base);
        const int trips = (n + G - 1) / G;
        for (int q = 0; q < trips; ++q) {
            const int k = q * G + grp;
            const uint32_t ck = __shfl_sync(0xffffffffu, c, k);
            const float vk = __shfl_sync(0xffffffffu, v, k);
            if (k < n && r != 0.0f) atomicAdd(bp + (uint64_t)ck * BT + b, __fmul_rn(vk, r));
        }
    }
}

__global__ void k_batch_update_zero(const float* __restrict__ norm, uint32_t cols, uint32_t BT,
                                    const uint32_t* __restrict__ remaining, float* __restrict__ f,
                                    float* __restrict__ bp) {
    const uint64_t n = (uint64_t)cols * BT;
    for (uint64_t o = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; o < n;
         o += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t c = (uint32_t)(o / BT), b = (uint32_t)(o % BT);
        const float acc = bp[o];
        bp[o] = 0.0f;
        if (remaining[b] > 0) {
            const float t = __fmul_rn(f[o], acc);
            const float nn = norm[c];
            f[o] = (nn == 0.0f) ? t : __fdiv_rn(t, nn);
        }
    }
}

__global__ void k_batch_tick(uint32_t* remaining, uint32_t BT) {
    if (threadIdx.x < BT && remaining[threadIdx.x] > 0) remaining[threadIdx.x] -= 1;
}

// Persistent batched MLEM: `steps` iterations of the tile in one cooperative
// launch (every block resident).  Per iteration: forward projection and
// correlation over all rows of A, grid barrier, back projection and update
// over all rows of Aᵀ for the slots with iterations left, grid barrier, tick
// of the per-slot counters by block 0.  The warps of the grid stride over
// row groups; each row is summed exactly as by k_batch_fp / k_batch_bp (same
// chains, same order), so an instance's bits do not depend on which kernel
// form runs it.
template <typename V, int W>
__global__ void __launch_bounds__(256, 6)
k_batch_loop(const uint64_t* __restrict__ rp, const uint32_t* __restrict__ ix, const V* __restrict__ vl,
             uint32_t rows, const uint64_t* __restrict__ rpT, const uint32_t* __restrict__ ixT,
             const V* __restrict__ vlT, uint32_t cols, const float* __restrict__ norm, uint32_t BT,
             uint32_t na, const int32_t* __restrict__ g, float* f, float* ratio, uint32_t* remaining, uint32_t steps,
             unsigned* count, int* err) {
    constexpr uint32_t RPW = 32 / W;  // rows per warp
    const int lane = threadIdx.x & 31, sl = lane % W;
    // 32-bit row counters (rows, cols < 2^32; a resident grid has < 2^16 warps)
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t stride = ((gridDim.x * blockDim.x) >> 5) * RPW;
    unsigned k = 0;
    for (uint32_t step = 0; step < steps; ++step) {
        for (uint32_t first = warp * RPW; first < rows; first += stride) {
            const uint32_t row = first + lane / W;
            const bool ok = row < rows;
            float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
            batch_rows<V, W, false>(rp, ix, vl, f, BT, na, row, ok, lane, acc);
            if (ok && sl < W / 4 && (uint32_t)sl * 4 < na) {
                const uint64_t o = (uint64_t)row * BT + sl * 4;
                const int4 gg = *reinterpret_cast<const int4*>(g + o);
                *reinterpret_cast<float4*>(ratio + o) = make_float4(correl1(gg.x, acc.x), correl1(gg.y, acc.y),
                                                                    correl1(gg.z, acc.z), correl1(gg.w, acc.w));
            }
        }
        if (!grid_barrier(count, ++k, err)) return;
        for (uint32_t first = warp * RPW; first < cols; first += stride) {
            const uint32_t c = first + lane / W;
            const bool ok = c < cols;
            float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
            batch_rows<V, W, false>(rpT, ixT, vlT, ratio, BT, na, c, ok, lane, acc);
            if (ok && sl < W / 4 && (uint32_t)sl * 4 < na) {
                const uint64_t o = (uint64_t)c * BT + sl * 4;
                const uint4 rem = *reinterpret_cast<const uint4*>(remaining + sl * 4);
                const float n = norm[c];
                float4 fv = *reinterpret_cast<const float4*>(f + o);
                if (rem.x) fv.x = update1(fv.x, acc.x, n);
                if (rem.y) fv.y = update1(fv.y, acc.y, n);
                if (rem.z) fv.z = update1(fv.z, acc.z, n);
                if (rem.w) fv.w = update1(fv.w, acc.w, n);
                *reinterpret_cast<float4*>(f + o) = fv;
            }
        }
        if (!grid_barrier(count, ++k, err)) return;
        // every block has read `remaining` for this iteration; the tick is seen
        // by the next back projection through the next barrier
        if (blockIdx.x == 0 && threadIdx.x < BT && remaining[threadIdx.x] > 0) remaining[threadIdx.x] -= 1;
    }
}

template <int W, typename V>
void fp_w(const DevCsr& A, const BatchArgs& b, L2Window win, cudaStream_t s) {
    launch_ex(k_batch_fp<V, W>, dim3(ceil_div_u((uint64_t)A.nrows * W, 256)), dim3(256), 0, s, win, A.rowptr,
              A.idx, static_cast<const V*>(A.val), (const float*)b.f, A.nrows, b.tile, b.slots(), b.g, b.ratio);
}

template <int W, typename V>
void bp_w(const DevCsr& AT, const float* norm, const BatchArgs& b, L2Window win, cudaStream_t s) {
    launch_ex(k_batch_bp<V, W>, dim3(ceil_div_u((uint64_t)AT.nrows * W, 256)), dim3(256), 0, s, win, AT.rowptr,
              AT.idx, static_cast<const V*>(AT.val), (const float*)b.ratio, AT.nrows, b.tile, b.slots(), norm,
              (const uint32_t*)b.remaining, b.f);
}

template <int BT, typename V>
void sc_bt(const DevCsr& A, const BatchArgs& b, float* bp, cudaStream_t s) {
    k_batch_scatter<V, BT><<<ceil_div_u((uint64_t)A.nrows * 32, 256), 256, 0, s>>>(
        A.rowptr, A.idx, static_cast<const V*>(A.val), b.ratio, A.nrows, bp);
    MLEM_LAUNCHED();
}

// Lanes per row for a launch of W slots: a matrix whose rows all fit the GPU at
// once with 8 lanes each (48 warps per SM) takes no fewer, since only the
// length of a row's chains counts there (1,770 rows, one iteration: 4 lanes 14.4,
// 8 lanes 12.4 us; 108,000 / 663,000 rows: 4 lanes 5% / 12% faster).
int row_lanes(uint32_t w, uint32_t rows) { return w == 4 && rows <= 152u * 48u * 4u ? 8 : (int)w; }

template <typename V>
void fp_v(const DevCsr& A, const BatchArgs& b, L2Window win, cudaStream_t s) {
    switch (row_lanes(b.width(), A.nrows)) {
        case 4: fp_w<4, V>(A, b, win, s); break;
        case 8: fp_w<8, V>(A, b, win, s); break;
        case 16: fp_w<16, V>(A, b, win, s); break;
        default: fp_w<32, V>(A, b, win, s);
    }
}
template <typename V>
void bp_v(const DevCsr& AT, const float* norm, const BatchArgs& b, L2Window win, cudaStream_t s) {
    switch (row_lanes(b.width(), AT.nrows)) {
        case 4: bp_w<4, V>(AT, norm, b, win, s); break;
        case 8: bp_w<8, V>(AT, norm, b, win, s); break;
        case 16: bp_w<16, V>(AT, norm, b, win, s); break;
        default: bp_w<32, V>(AT, norm, b, win, s);
    }
}
template <typename V>
void sc_v(const DevCsr& A, const BatchArgs& b, float* bp, cudaStream_t s) {
    if (b.tile == 32) sc_bt<32, V>(A, b, bp, s);
    else if (b.tile == 16) sc_bt<16, V>(A, b, bp, s);
    else sc_bt<8, V>(A, b, bp, s);
}

__global__ void k_slot_put(int32_t* __restrict__ G, float* __restrict__ F, uint32_t rows,
                           uint32_t cols, uint32_t BT, uint32_t b, const int32_t* __restrict__ g,
                           float init, const float* __restrict__ f0, uint32_t* __restrict__ remaining,
                           uint32_t iters, const uint32_t* __restrict__ lor_of, const uint32_t* __restrict__ vox_of) {
    const uint32_t n = rows > cols ? rows : cols;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        if (i < rows) G[(uint64_t)i * BT + b] = g[lor_of ? lor_of[i] : i];
        if (i < cols) F[(uint64_t)i * BT + b] = f0 ? f0[vox_of ? vox_of[i] : i] : init;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) remaining[b] = iters;
}

__global__ void k_slot_get(const float* __restrict__ F, uint32_t cols, uint32_t BT, uint32_t b,
                           float* __restrict__ out, const uint32_t* __restrict__ vox_of) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < cols; i += gridDim.x * blockDim.x)
        out[vox_of ? vox_of[i] : i] = F[(uint64_t)i * BT + b];
}

}  // namespace

void launch_slot_put(int32_t* G, float* F, uint32_t rows, uint32_t cols, uint32_t BT, uint32_t b,
                     const int32_t* g, float init, const float* f0, uint32_t* remaining,
                     uint32_t iters, const uint32_t* lor_of, const uint32_t* vox_of, cudaStream_t s) {
    const uint32_t n = std::max(rows, cols);
    const unsigned grid = std::max(1u, std::min<unsigned>(ceil_div_u(n, 256), 152u * 8u));
    k_slot_put<<<grid, 256, 0, s>>>(G, F, rows, cols, BT, b, g, init, f0, remaining, iters, lor_of, vox_of);
    MLEM_LAUNCHED();
}

void launch_slot_get(const float* F, uint32_t cols, uint32_t BT, uint32_t b, float* out,
                     const uint32_t* vox_of, cudaStream_t s) {
    const unsigned grid = std::max(1u, std::min<unsigned>(ceil_div_u(cols, 256), 152u * 8u));
    k_slot_get<<<grid, 256, 0, s>>>(F, cols, BT, b, out, vox_of);
    MLEM_LAUNCHED();
}

void launch_batch_fp(const DevCsr& A, const BatchArgs& b, L2Window win, cudaStream_t s) {
    if (A.nrows == 0) return;
    switch (A.vt) {
        case MLEM_VAL_F32: fp_v<float>(A, b, win, s); break;
        case MLEM_VAL_F16: fp_v<__half>(A, b, win, s); break;
        default: fp_v<__nv_bfloat16>(A, b, win, s);
    }
}

void launch_batch_bp_update(const DevCsr& AT, const float* norm, const BatchArgs& b, L2Window win,
                            cudaStream_t s) {
    if (AT.nrows == 0) return;
    switch (AT.vt) {
        case MLEM_VAL_F32: bp_v<float>(AT, norm, b, win, s); break;
        case MLEM_VAL_F16: bp_v<__half>(AT, norm, b, win, s); break;
        default: bp_v<__nv_bfloat16>(AT, norm, b, win, s);
    }
}

namespace {

template <typename V, int W>
void loop_w(const DevCsr& A, const DevCsr& AT, const float* norm, const BatchArgs& b, uint32_t steps,
            unsigned* count, int* err, cudaStream_t s) {
    auto kern = k_batch_loop<V, W>;
    // one resident wave: every block must be on the GPU at once for the barriers
    static const int bps = [kern] {
        int b = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kern, 256, 0) != cudaSuccess) {
            cudaGetLastError();
            b = 0;
        }
        return b;
    }();
    int dev = 0, sms = 0;
    MLEM_CUDA(cudaGetDevice(&dev));
    MLEM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    MLEM_REQUIRE(bps >= 1, MLEM_EUNSUPPORTED, "persistent batch kernel does not fit on an SM");
    MLEM_CUDA(cudaMemsetAsync(count, 0, sizeof(unsigned), s));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(bps * sms));
    cfg.blockDim = dim3(256);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    MLEM_CUDA(cudaLaunchKernelEx(&cfg, kern, (const uint64_t*)A.rowptr, (const uint32_t*)A.idx,
                                 static_cast<const V*>(A.val), A.nrows, (const uint64_t*)AT.rowptr,
                                 (const uint32_t*)AT.idx, static_cast<const V*>(AT.val), AT.nrows, norm, b.tile,
                                 b.slots(), b.g, b.f, b.ratio, b.remaining, steps, count, err));
    count_launch();
}

template <typename V>
void loop_v(const DevCsr& A, const DevCsr& AT, const float* norm, const BatchArgs& b, uint32_t steps,
            unsigned* count, int* err, cudaStream_t s) {
    switch (b.width()) {
        case 4: loop_w<V, 4>(A, AT, norm, b, steps, count, err, s); break;
        case 8: loop_w<V, 8>(A, AT, norm, b, steps, count, err, s); break;
        case 16: loop_w<V, 16>(A, AT, norm, b, steps, count, err, s); break;
        default: loop_w<V, 32>(A, AT, norm, b, steps, count, err, s);
    }
}

}  // namespace

void launch_batch_loop(const DevCsr& A, const DevCsr& AT, const float* norm, const BatchArgs& b, uint32_t steps,
                       unsigned* count, int* err, cudaStream_t s) {
    if (steps == 0 || A.nrows == 0) return;
    switch (A.vt) {
        case MLEM_VAL_F32: loop_v<float>(A, AT, norm, b, steps, count, err, s); break;
        case MLEM_VAL_F16: loop_v<__half>(A, AT, norm, b, steps, count, err, s); break;
        default: loop_v<__nv_bfloat16>(A, AT, norm, b, steps, count, err, s);
    }
}

void launch_batch_tick(const BatchArgs& b, cudaStream_t s) {
    k_batch_tick<<<1, 32, 0, s>>>(b.remaining, b.tile);
    MLEM_LAUNCHED();
}

void launch_batch_scatter(const DevCsr& A, const BatchArgs& b, float* bp, cudaStream_t s) {
    if (A.nrows == 0) return;
    switch (A.vt) {
        case MLEM_VAL_F32: sc_v<float>(A, b, bp, s); break;
        case MLEM_VAL_F16: sc_v<__half>(A, b, bp, s); break;
        default: sc_v<__nv_bfloat16>(A, b, bp, s);
    }
}

void launch_batch_update_zero(const float* norm, uint32_t cols, const BatchArgs& b, float* bp,
                              cudaStream_t s) {
    const uint64_t n = (uint64_t)cols * b.tile;
    if (n == 0) return;
    const unsigned grid = std::max(1u, std::min<unsigned>(ceil_div_u(n, 256), 152u * 16u));
    k_batch_update_zero<<<grid, 256, 0, s>>>(norm, cols, b.tile, b.remaining, b.f, bp);
    MLEM_LAUNCHED();
}

}  // namespace mlem
