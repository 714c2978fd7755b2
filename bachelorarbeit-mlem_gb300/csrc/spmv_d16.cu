// spmv_d16.cu — projections over 16-bit delta-coded column indices (D16).
//
// A row is cut into steps of 8·L entries, L = op.d16_lanes (4 or 8) lanes per
// row: position p of a row belongs to lane p % L as element p / L of that
// lane's sequence, so one gather instruction covers L consecutive entries of
// the row (few cache lines: its columns are ascending and close).  Each entry
// stores the difference between its column and the column L positions earlier
// (the previous element of the same lane; the row's first column for the first
// L positions): every lane decodes its own columns with one add per entry, no
// scans and no shuffles.  Layout of an operand in D16 form (beside the u32 CSR):
//   dvptr[r]  first 8-entry vector of row r (u64[nrows + 1]); vector
//             dvptr[r] + k·L + l holds lane l's elements 8k..8k+7
//   dbase[r]  first column of row r
//   d16[8 v + j], dval[8 v + j]  the delta and the value (the operand's type)
// A difference of 65,536 or more is bridged by dummy entries (column = the
// earlier column + 65,535) and rows are padded to whole steps with delta 0;
// both carry the value -0.0, which no stored entry has (a stored -0.0 becomes
// +0.0).  A row whose sum is NaN is summed again without them, so that an
// infinite or NaN element of x that the row does not list stays out of its sum.
//
// What bounds it: the bytes of the stream, (2 + value) per position.  Dummies
// and padding add 8% (A) and 14% (A^T) on the 3-D mid matrix, 9% and 16% on
// the 12 GB class.  Measured and not kept: a half step (4 entries per lane) at
// a row's end, 4% / 7% of padding but rows that start inside a 128-byte line
// (mid, FP32 / FP16 values: 0.442 / 0.361 ms per iteration against 0.431 /
// 0.313).  The lane sums (kSums chains per lane) are reduced by a fixed xor
// tree: deterministic.
#include "kernels.cuh"

#include <algorithm>
#include <cstring>
#include <vector>

namespace mlem {

namespace {

template <typename V>
struct Val8;

template <>
struct Val8<float> {
    static __device__ __forceinline__ void load(const float* p, uint64_t v, float out[8]) {
        const float4* q = reinterpret_cast<const float4*>(p) + 2 * v;
        const float4 a = ld_stream(q), b = ld_stream(q + 1);
        out[0] = a.x; out[1] = a.y; out[2] = a.z; out[3] = a.w;
        out[4] = b.x; out[5] = b.y; out[6] = b.z; out[7] = b.w;
    }
};

template <>
struct Val8<__half> {
    static __device__ __forceinline__ void load(const __half* p, uint64_t v, float out[8]) {
        const uint4 u = ld_stream(reinterpret_cast<const uint4*>(p) + v);
        const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[k]));
            out[2 * k] = f.x;
            out[2 * k + 1] = f.y;
        }
    }
};

template <>
struct Val8<__nv_bfloat16> {
    static __device__ __forceinline__ void load(const __nv_bfloat16* p, uint64_t v, float out[8]) {
        const uint4 u = ld_stream(reinterpret_cast<const uint4*>(p) + v);
        const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w[k]));
            out[2 * k] = f.x;
            out[2 * k + 1] = f.y;
        }
    }
};

// The row of this thread's group of L lanes (threads may outnumber 2^32).
template <int L>
__device__ __forceinline__ uint32_t group_row() { return blockIdx.x * (blockDim.x / L) + threadIdx.x / L; }

// The value of dummies and padding.
template <typename V>
__device__ __forceinline__ V pad_value() {
    V v;
    *reinterpret_cast<uint16_t*>(&v) = 0x8000u;
    return v;
}
template <>
__device__ __forceinline__ float pad_value<float>() { return -0.0f; }

// Sums per lane: element j of a lane's vector goes to sum j mod kSums, 16 chains
// per row as with 16 lanes of one sum each.
template <int LPR>
constexpr int kSums = 16 / LPR;

template <int LPR>
__device__ __forceinline__ float lane_sum(const float* acc) {
    return kSums<LPR> == 4 ? (acc[0] + acc[1]) + (acc[2] + acc[kSums<LPR> - 1]) : acc[0] + acc[1];
}

// A row's sum again, in the same order, without the dummies and the padding, by
// one thread: for rows whose sum is NaN (see the head of the file).  It ends as
// soon as a lane's sum is NaN, as the row's then is: where the image holds NaN,
// after a few entries.  An iteration of the 12 GB class on an image of NaN 2.99 ms
// (FP16 values 2.31), walking every row to its end 29.3 (29.5); on an ordinary
// image 2.79 (2.04).  Measured and not kept: by the row's group of lanes, which
// needs no early end, but the call costs ordinary images 2% with FP16 values.
template <typename V, int LPR>
__device__ __noinline__ float d16_row_real(const uint64_t* __restrict__ dvptr, const uint32_t* __restrict__ dbase,
                                           const uint16_t* __restrict__ d16, const V* __restrict__ dval,
                                           const float* __restrict__ x, uint32_t row) {
    const uint64_t v0 = dvptr[row], v1 = dvptr[row + 1];
    float sum[LPR];
    for (int l = 0; l < LPR; ++l) {
        uint32_t col = dbase[row];
        float acc[kSums<LPR>] = {};
        for (uint64_t v = v0 + l; v < v1; v += LPR) {
            for (int j = 0; j < 8; ++j) {
                col += d16[8 * v + j];
                const float a = (float)dval[8 * v + j];
                if (__float_as_uint(a) != 0x80000000u) acc[j % kSums<LPR>] = fmaf(a, ld_after(x + col), acc[j % kSums<LPR>]);
            }
            if (isnan(lane_sum<LPR>(acc))) return lane_sum<LPR>(acc);  // as it will be whatever follows
        }
        sum[l] = lane_sum<LPR>(acc);
    }
    for (int o = LPR / 2; o > 0; o >>= 1)
        for (int l = 0; l < o; ++l) sum[l] += sum[l + o];
    return sum[0];
}

// N steps of a lane: loads, columns, gathers, FMAs.  dp, vp: the lane's delta and
// value vector of the first.
template <typename V, int LPR, int N>
__device__ __forceinline__ void d16_steps(const uint4* dp, const V* vp, const float* __restrict__ x, uint32_t& prev,
                                          float (&acc)[kSums<LPR>]) {
    uint4 dw[N];
    float a[N][8];
#pragma unroll
    for (int u = 0; u < N; ++u) {
        dw[u] = ld_stream(dp + u * LPR);
        Val8<V>::load(vp, (uint64_t)u * LPR, a[u]);
    }
    uint32_t col[N][8];
#pragma unroll
    for (int u = 0; u < N; ++u) {
        const uint32_t w[4] = {dw[u].x, dw[u].y, dw[u].z, dw[u].w};
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            prev += (w[j >> 1] >> (16 * (j & 1))) & 0xFFFFu;
            col[u][j] = prev;
        }
    }
    float gx[N][8];
#pragma unroll
    for (int u = 0; u < N; ++u)
#pragma unroll
        for (int j = 0; j < 8; ++j) gx[u][j] = ld_after(x + col[u][j]);
#pragma unroll
    for (int u = 0; u < N; ++u)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j % kSums<LPR>] = fmaf(a[u][j], gx[u][j], acc[j % kSums<LPR>]);
}

// A stretch of whole vectors into L2 ahead of the loads.
__device__ __forceinline__ void d16_prefetch(const void* p, uint64_t bytes) {
    const uint64_t a = reinterpret_cast<uint64_t>(p);
    for (uint64_t q = 0; q < bytes; q += 65536)
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a + q),
                     "r"((uint32_t)(bytes - q < 65536 ? bytes - q : 65536)) : "memory");
}

// The sum of a row of `nsteps` steps by its group of LPR lanes (vp, dp: the row's
// first vectors, col: its first column).
template <typename V, int LPR, int U>
__device__ __forceinline__ float d16_row(const uint4* dp, const V* vp, const float* __restrict__ x, uint32_t col,
                                         uint32_t nsteps, uint32_t gl) {
    uint32_t prev = col;  // column of this lane's previous element
    float acc[kSums<LPR>] = {};
    dp += gl;
    vp += 8 * gl;
    uint32_t k = 0;
    for (; k + U <= nsteps; k += U) {
        d16_steps<V, LPR, U>(dp, vp, x, prev, acc);
        dp += U * LPR;
        vp += U * 8 * LPR;
    }
    if (U == 2 && k < nsteps) d16_steps<V, LPR, 1>(dp, vp, x, prev, acc);
    return lane_sum<LPR>(acc);
}

template <int EPI>
__device__ __forceinline__ void d16_epi(uint32_t row, float acc, const int32_t* __restrict__ g, float* __restrict__ out,
                                        float* __restrict__ fwproj, float* __restrict__ f,
                                        const float* __restrict__ norm) {
    if (EPI == (int)Epi::Correl) {
        out[row] = (acc != 0.0f) ? __fdiv_rn((float)ld_after(g + row), acc) : 0.0f;
        if (fwproj) fwproj[row] = acc;
    } else if (EPI == (int)Epi::Update) {
        const float tt = __fmul_rn(f[row], acc);
        const float nn = norm[row];
        f[row] = (nn == 0.0f) ? tt : __fdiv_rn(tt, nn);
    } else {
        out[row] = acc;
    }
}

// Blocks per SM, measured on the 3-D mid / 12 GB-class matrix, ms per iteration
// with U = 1 and U = 2: FP32 values 5 blocks (48 registers) 0.431, 0.433 / 2.83,
// 2.90, 8 and 6 blocks 0.472, 0.438 / 3.77, 2.99; FP16 values 8 and 6 blocks (32
// and 40 registers) 0.313, 0.316 / 2.14, 2.04, 5 blocks 0.335, 0.337 / 2.08, 2.09.
template <typename V, int EPI, int LPR, int U>
__global__ void __launch_bounds__(256, sizeof(V) == 4 ? 5 : U == 2 ? 6 : 8)
k_csr_d16(const uint64_t* __restrict__ dvptr, const uint32_t* __restrict__ dbase, const uint16_t* __restrict__ d16,
          const V* __restrict__ dval, const float* __restrict__ x, uint32_t nrows, const int32_t* __restrict__ g,
          float* __restrict__ out, float* __restrict__ fwproj, float* __restrict__ f, const float* __restrict__ norm) {
    grid_release();
    const uint32_t row = group_row<LPR>();
    const uint32_t gl = threadIdx.x % LPR;
    const bool live = row < nrows;
    const uint64_t v0 = live ? dvptr[row] : 0, v1 = live ? dvptr[row + 1] : 0;
    const uint32_t nsteps = (uint32_t)((v1 - v0) / LPR);
    const uint4* dp = reinterpret_cast<const uint4*>(d16) + v0;
    const V* vp = dval + 8 * v0;
    if (live && gl == 0 && v1 > v0) {
        d16_prefetch(dp, 16 * (v1 - v0));
        d16_prefetch(vp, 8 * sizeof(V) * (v1 - v0));
    }
    const uint32_t col = live ? dbase[row] : 0u;
    grid_wait();
    float acc = d16_row<V, LPR, U>(dp, vp, x, col, nsteps, gl);
#pragma unroll
    for (int o = LPR / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o, LPR);
    if (live && gl == 0) {
        if (isnan(acc)) acc = d16_row_real<V, LPR>(dvptr, dbase, d16, dval, x, row);
        d16_epi<EPI>(row, acc, g, out, fwproj, f, norm);
    }
}

// The same sums over the merge-path tiles of whole rows (merge.cu): a block of
// 128 threads lists the tile's rows that have entries, writes the empty ones
// there and then, and its lane groups take the listed rows in turn.  The
// tile's vectors are one stretch of the copy, prefetched at once.  An iteration
// of the 3-D mid matrix over the CSR arrays and over the copy: 0.677 / 0.556 ms in
// natural order, 0.603 / 0.452 ms in the locality layout (rows in order, without
// tiles: 0.467 / 0.423 ms).
constexpr uint32_t kTileT = 128;

template <typename V, int EPI, int LPR, int U>
__global__ void __launch_bounds__(kTileT, sizeof(V) == 4 ? 10 : 12)
k_merge_d16(const uint32_t* __restrict__ ti, const uint64_t* __restrict__ dvptr, const uint32_t* __restrict__ dbase,
            const uint16_t* __restrict__ d16, const V* __restrict__ dval, const float* __restrict__ x,
            const int32_t* __restrict__ g, float* __restrict__ out, float* __restrict__ fwproj, float* __restrict__ f,
            const float* __restrict__ norm) {
    grid_release();
    const uint32_t I0 = ti[blockIdx.x], nrow = ti[blockIdx.x + 1] - I0;
    __shared__ uint32_t s_row[kTileT], s_at[kTileT], s_steps[kTileT], s_cnt[kTileT / 32];
    const uint32_t w = threadIdx.x >> 5, lane = threadIdx.x & 31, grp = threadIdx.x / LPR, gl = threadIdx.x % LPR;
    const unsigned mask = ((1u << LPR) - 1u) << (lane & ~(LPR - 1));
    const uint64_t V0 = dvptr[I0];
    if (threadIdx.x == 0) {
        const uint64_t nv = dvptr[I0 + nrow] - V0;
        d16_prefetch(d16 + 8 * V0, 16 * nv);
        d16_prefetch(dval + 8 * V0, 8 * sizeof(V) * nv);
    }
    if (nrow == 0) grid_wait();  // every block waits before it ends
    for (uint32_t c0 = 0; c0 < nrow; c0 += kTileT) {
        const uint32_t i = c0 + threadIdx.x;
        const bool live = i < nrow;
        const uint64_t a = live ? dvptr[I0 + i] : 0, b = live ? dvptr[I0 + i + 1] : 0;
        if (c0 == 0) grid_wait();
        const bool keep = a < b;
        if (live && !keep) d16_epi<EPI>(I0 + i, 0.f, g, out, fwproj, f, norm);
        const unsigned kept = __ballot_sync(0xffffffffu, keep);
        if (c0) __syncthreads();  // the list of the previous rows is used up
        if (lane == 0) s_cnt[w] = __popc(kept);
        __syncthreads();
        uint32_t n = 0, at = __popc(kept & ((1u << lane) - 1u));
#pragma unroll
        for (uint32_t q = 0; q < kTileT / 32; ++q) {
            if (q == w) at += n;
            n += s_cnt[q];
        }
        if (keep) {
            s_row[at] = I0 + i;
            s_at[at] = (uint32_t)(a - V0);
            s_steps[at] = (uint32_t)((b - a) / LPR);
        }
        __syncthreads();
        for (uint32_t j = grp; j < n; j += kTileT / LPR) {
            const uint32_t row = s_row[j];
            const uint64_t v = V0 + s_at[j];
            float acc = d16_row<V, LPR, U>(reinterpret_cast<const uint4*>(d16) + v, dval + 8 * v, x, dbase[row],
                                           s_steps[j], gl);
#pragma unroll
            for (int o = LPR / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(mask, acc, o, LPR);
            if (gl == 0) {
                if (isnan(acc)) acc = d16_row_real<V, LPR>(dvptr, dbase, d16, dval, x, row);
                d16_epi<EPI>(row, acc, g, out, fwproj, f, norm);
            }
        }
    }
}

// ---------------------------------------------------------------- conversion
// Sets *unsorted when some row lists a column below its predecessor.
__global__ void k_d16_check(const uint64_t* __restrict__ rowptr, const uint32_t* __restrict__ col, uint32_t rows,
                            int* __restrict__ unsorted) {
    const int lane = threadIdx.x & 31;
    const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < rows; r += nw) {
        const uint64_t s = rowptr[r], t = rowptr[r + 1];
        bool bad = false;
        for (uint64_t e = s + 1 + lane; e < t; e += 32) bad |= col[e] < col[e - 1];
        if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(unsorted, 1);
    }
}

// One slice (L consecutive positions, one per lane) of a row's walk by its
// group of L lanes: lane i's position takes the next entry unless its column
// lies 65,536 or more past `ring`, the column L positions earlier, when it
// takes a dummy.  e = next entry on entry and on return; ent = the lane's
// entry, ~0 for a dummy or padding; returns the lane's delta.
template <int L>
__device__ __forceinline__ uint32_t d16_slice(const uint32_t* __restrict__ col, uint64_t t, uint64_t& e, uint32_t& ring,
                                              uint64_t& ent, unsigned mask, int gl) {
    const bool have = e + gl < t;
    const uint32_t c = have ? col[e + gl] : ring;
    if (!__any_sync(mask, c - ring >= 65536u)) {
        const uint32_t d = c - ring;
        ent = have ? e + gl : ~0ull;
        ring = c;
        e += L;
        return d;
    }
    uint32_t d = 0;
    ent = ~0ull;
#pragma unroll 1
    for (int i = 0; i < L; ++i) {
        const uint32_t r = __shfl_sync(mask, ring, i, L);
        if (e >= t) break;
        const uint32_t ci = col[e];
        const bool dummy = ci - r >= 65536u;
        if (gl == i) {
            d = dummy ? 65535u : ci - r;
            ent = dummy ? ~0ull : e;
            ring = r + d;
        }
        if (!dummy) ++e;
    }
    return d;
}

__device__ __forceinline__ unsigned group_mask(int L) { return ((1u << L) - 1u) << ((threadIdx.x & 31) & ~(L - 1)); }

// Vectors per row (positions rounded up to whole steps of 8·L).  L lanes per row.
// *sparse sums the vectors of the rows that hold more than twice their entries
// (and a step); once they alone are above max_vec no further row is walked, so
// that an operand that will not get a copy costs no long walks over dummies.
template <int L>
__global__ void __launch_bounds__(256)
k_d16_count(const uint64_t* __restrict__ rowptr, const uint32_t* __restrict__ col, uint32_t rows,
            uint32_t* __restrict__ nvec, uint64_t max_vec, unsigned long long* sparse) {
    const uint32_t r = group_row<L>();
    const int gl = threadIdx.x % L;
    if (r >= rows) return;  // whole group
    const unsigned mask = group_mask(L);
    uint64_t e = rowptr[r], ent;
    const uint64_t t = rowptr[r + 1], len = t - e;
    const bool over = __shfl_sync(mask, *(volatile unsigned long long*)sparse, 0, L) > max_vec;
    uint32_t n = 0, ring = e < t ? col[e] : 0u;
    if (!over)
        for (; e < t; ++n) d16_slice<L>(col, t, e, ring, ent, mask, gl);
    n = (n + 7) / 8 * L;
    if (gl == 0) {
        nvec[r] = n;
        if (n > L && n / 2 > (len + 7) / 8) atomicAdd(sparse, (unsigned long long)n);
    }
}

// Deltas and values at their positions, padding included.  L lanes per row; a
// lane collects its 8 elements of a step in shared memory and writes them as
// 16-byte vectors (both copies of the mid matrix: 5 ms, against 45 ms with one
// thread per row and one store per entry).
template <typename V, int L>
__global__ void __launch_bounds__(256)
k_d16_fill(const uint64_t* __restrict__ rowptr, const uint32_t* __restrict__ col, const V* __restrict__ val,
           uint32_t rows, const uint64_t* __restrict__ dvptr, uint32_t* __restrict__ dbase,
           uint16_t* __restrict__ d16, V* __restrict__ dval) {
    __shared__ __align__(16) uint16_t sd[256][8];
    __shared__ __align__(16) V sv[256][8];
    const uint32_t r = group_row<L>();
    const int gl = threadIdx.x % L;
    if (r >= rows) return;  // whole group
    const unsigned mask = group_mask(L);
    uint64_t e = rowptr[r];
    const uint64_t t = rowptr[r + 1], v1 = dvptr[r + 1];
    uint32_t ring = e < t ? col[e] : 0u;
    if (gl == 0) dbase[r] = ring;
    uint16_t* md = sd[threadIdx.x];
    V* mv = sv[threadIdx.x];
    for (uint64_t v = dvptr[r]; v < v1; v += L) {
        for (int j = 0; j < 8; ++j) {
            uint64_t ent = ~0ull;
            uint32_t d = 0;
            if (e < t) d = d16_slice<L>(col, t, e, ring, ent, mask, gl);
            V a = pad_value<V>();
            if (ent != ~0ull) a = (float)val[ent] == 0.0f ? (V)0.0f : val[ent];
            md[j] = (uint16_t)d;
            mv[j] = a;
        }
        reinterpret_cast<uint4*>(d16)[v + gl] = *reinterpret_cast<const uint4*>(md);
#pragma unroll
        for (int i = 0; i < (int)sizeof(V) / 2; ++i)
            reinterpret_cast<uint4*>(dval + 8 * (v + gl))[i] = reinterpret_cast<const uint4*>(mv)[i];
    }
}

unsigned grid_rows(uint32_t rows) {
    return std::max(1u, std::min<unsigned>(ceil_div_u((uint64_t)rows * 32, 256), 152u * 32u));
}

unsigned grid_groups(uint32_t rows, int lanes) { return ceil_div_u((uint64_t)rows * lanes, 256); }

template <typename V>
void d16_fill(DevCsr& op, const uint32_t* idx, const void* val, cudaStream_t s) {
    if (op.d16_lanes == 4)
        k_d16_fill<V, 4><<<grid_groups(op.nrows, 4), 256, 0, s>>>(op.rowptr, idx, static_cast<const V*>(val), op.nrows,
                                                                  op.dvptr, op.dbase, op.d16, static_cast<V*>(op.dval));
    else
        k_d16_fill<V, 8><<<grid_groups(op.nrows, 8), 256, 0, s>>>(op.rowptr, idx, static_cast<const V*>(val), op.nrows,
                                                                  op.dvptr, op.dbase, op.d16, static_cast<V*>(op.dval));
    MLEM_LAUNCHED();
}

// A copy of the operand's entries with every row sorted by column (stable),
// made on the host: only for rows given out of order (generated and
// transposed operands are sorted already).
void sorted_copy(const DevCsr& op, uint32_t*& idx, void*& val, cudaStream_t s) {
    const size_t vb = val_bytes(op.vt);
    std::vector<uint64_t> rp(op.nrows + 1);
    std::vector<uint32_t> c(op.nnz);
    std::vector<unsigned char> v(op.nnz * vb);
    MLEM_CUDA(cudaMemcpyAsync(rp.data(), op.rowptr, sizeof(uint64_t) * rp.size(), cudaMemcpyDeviceToHost, s));
    MLEM_CUDA(cudaMemcpyAsync(c.data(), op.idx, sizeof(uint32_t) * op.nnz, cudaMemcpyDeviceToHost, s));
    MLEM_CUDA(cudaMemcpyAsync(v.data(), op.val, vb * op.nnz, cudaMemcpyDeviceToHost, s));
    MLEM_CUDA(cudaStreamSynchronize(s));
    std::vector<uint32_t> c2(op.nnz);
    std::vector<unsigned char> v2(op.nnz * vb);
#pragma omp parallel
    {
        std::vector<uint64_t> perm;
#pragma omp for schedule(dynamic, 64)
        for (int64_t r = 0; r < (int64_t)op.nrows; ++r) {
            const uint64_t a = rp[r], b = rp[r + 1];
            perm.resize(b - a);
            for (uint64_t e = a; e < b; ++e) perm[e - a] = e;
            std::stable_sort(perm.begin(), perm.end(), [&](uint64_t x, uint64_t y) { return c[x] < c[y]; });
            for (uint64_t k = 0; k < b - a; ++k) {
                c2[a + k] = c[perm[k]];
                std::memcpy(&v2[(a + k) * vb], &v[perm[k] * vb], vb);
            }
        }
    }
    MLEM_CUDA(cudaMalloc(&idx, sizeof(uint32_t) * std::max<uint64_t>(op.nnz, 1)));
    MLEM_CUDA(cudaMalloc(&val, vb * std::max<uint64_t>(op.nnz, 1)));
    MLEM_CUDA(cudaMemcpyAsync(idx, c2.data(), sizeof(uint32_t) * op.nnz, cudaMemcpyHostToDevice, s));
    MLEM_CUDA(cudaMemcpyAsync(val, v2.data(), vb * op.nnz, cudaMemcpyHostToDevice, s));
    MLEM_CUDA(cudaStreamSynchronize(s));
}

// tiles: first rows of the merge-path tiles (device) or null for rows in order.
struct Tiles {
    const uint32_t* first = nullptr;
    uint64_t n = 0;
};

template <typename V, int EPI, int LPR, int U>
void d16_launch(const DevCsr& op, Tiles t, const float* x, const EpiArgs& e, L2Window win, cudaStream_t s) {
    const V* dval = static_cast<const V*>(op.dval);
    if (t.first)
        launch_attrs(e.overlap, k_merge_d16<V, EPI, LPR, U>, dim3((unsigned)t.n), dim3(kTileT), 0, s, win, t.first,
                     op.dvptr, op.dbase, op.d16, dval, x, e.g, e.out, e.fwproj, e.f, e.norm);
    else
        launch_attrs(e.overlap, k_csr_d16<V, EPI, LPR, U>, dim3(grid_groups(op.nrows, LPR)), dim3(256), 0, s, win,
                     op.dvptr, op.dbase, op.d16, dval, x, op.nrows, e.g, e.out, e.fwproj, e.f, e.norm);
}

template <typename V, int EPI>
void d16_shape(const DevCsr& op, Tiles t, const float* x, const EpiArgs& e, int unroll, L2Window win, cudaStream_t s) {
    if (op.d16_lanes == 4) {
        if (unroll >= 2) d16_launch<V, EPI, 4, 2>(op, t, x, e, win, s);
        else d16_launch<V, EPI, 4, 1>(op, t, x, e, win, s);
    } else {
        if (unroll >= 2) d16_launch<V, EPI, 8, 2>(op, t, x, e, win, s);
        else d16_launch<V, EPI, 8, 1>(op, t, x, e, win, s);
    }
}

template <typename V>
void d16_epilogue(const DevCsr& op, Tiles t, const float* x, const EpiArgs& e, int unroll, L2Window win,
                  cudaStream_t s) {
    switch (e.kind) {
        case Epi::Correl: d16_shape<V, (int)Epi::Correl>(op, t, x, e, unroll, win, s); break;
        case Epi::Update: d16_shape<V, (int)Epi::Update>(op, t, x, e, unroll, win, s); break;
        default: d16_shape<V, (int)Epi::Raw>(op, t, x, e, unroll, win, s);
    }
}

void d16_dispatch(const DevCsr& op, Tiles t, const float* x, const EpiArgs& e, int unroll, L2Window win,
                  cudaStream_t s) {
    MLEM_REQUIRE(op.d16 != nullptr, MLEM_EINVAL, "operand has no D16 indices");
    switch (op.vt) {
        case MLEM_VAL_F32: d16_epilogue<float>(op, t, x, e, unroll, win, s); break;
        case MLEM_VAL_F16: d16_epilogue<__half>(op, t, x, e, unroll, win, s); break;
        default: d16_epilogue<__nv_bfloat16>(op, t, x, e, unroll, win, s);
    }
}

}  // namespace

void free_d16(DevCsr& op) {
    cudaFree(op.dvptr);
    cudaFree(op.dbase);
    cudaFree(op.d16);
    cudaFree(op.dval);
    op.dvptr = nullptr;
    op.dbase = nullptr;
    op.d16 = nullptr;
    op.dval = nullptr;
    op.dvec = 0;
    op.d16_lanes = 0;
}

bool build_d16(DevCsr& op, bool sort_rows, uint64_t max_bytes, cudaStream_t s) {
    const uint64_t per_vec = 8 * (sizeof(uint16_t) + val_bytes(op.vt)), per_row = 12ull * op.nrows + 8;
    if (per_row >= max_bytes) return false;
    const uint64_t max_vec = (max_bytes - per_row) / per_vec;
    const uint64_t R = std::max<uint32_t>(op.nrows, 1);
    // 8 lanes per row cover more neighbouring columns per gather, 4 pad short
    // rows less (steps of 64 or 32 entries)
    const int lanes = op.nrows && op.nnz / op.nrows >= kD16LongRow ? 8 : 4;
    // deltas need every row in ascending column order
    const uint32_t* idx = op.idx;
    const void* val = op.val;
    uint32_t* sidx = nullptr;
    void* sval = nullptr;
    uint32_t* nvec = nullptr;
    unsigned long long* word = nullptr;  // [0] k_d16_check's flag, [1] k_d16_count's sum
    int unsorted = 0;
    bool fits = true;
    try {
        MLEM_CUDA(cudaMallocAsync(&word, 16, s));
        MLEM_CUDA(cudaMemsetAsync(word, 0, 16, s));
        if (op.nrows) {
            k_d16_check<<<grid_rows(op.nrows), 256, 0, s>>>(op.rowptr, op.idx, op.nrows, reinterpret_cast<int*>(word));
            MLEM_LAUNCHED();
        }
        MLEM_CUDA(cudaMemcpyAsync(&unsorted, word, sizeof(int), cudaMemcpyDeviceToHost, s));
        MLEM_CUDA(cudaStreamSynchronize(s));
        if (unsorted && !sort_rows) {
            cudaFreeAsync(word, s);
            return false;
        }
        if (unsorted) {
            sorted_copy(op, sidx, sval, s);
            idx = sidx;
            val = sval;
        }
        op.d16_lanes = lanes;
        MLEM_CUDA(cudaMallocAsync(&nvec, sizeof(uint32_t) * R, s));
        MLEM_CUDA(cudaMalloc(&op.dvptr, sizeof(uint64_t) * (R + 1)));
        if (op.nrows) {
            if (lanes == 4)
                k_d16_count<4><<<grid_groups(op.nrows, 4), 256, 0, s>>>(op.rowptr, idx, op.nrows, nvec, max_vec, word + 1);
            else
                k_d16_count<8><<<grid_groups(op.nrows, 8), 256, 0, s>>>(op.rowptr, idx, op.nrows, nvec, max_vec, word + 1);
            MLEM_LAUNCHED();
        }
        scan_counts_u64(nvec, op.dvptr, op.nrows, s);
        uint64_t nv = 0, sparse = 0;
        MLEM_CUDA(cudaMemcpyAsync(&nv, op.dvptr + op.nrows, sizeof(uint64_t), cudaMemcpyDeviceToHost, s));
        MLEM_CUDA(cudaMemcpyAsync(&sparse, word + 1, sizeof(uint64_t), cudaMemcpyDeviceToHost, s));
        MLEM_CUDA(cudaStreamSynchronize(s));
        fits = std::max(nv, sparse) <= max_vec;
        const uint64_t slots = 8 * std::max<uint64_t>(nv, 1);
        if (fits) {
            op.dvec = nv;
            MLEM_CUDA(cudaMalloc(&op.dbase, sizeof(uint32_t) * R));
            MLEM_CUDA(cudaMalloc(&op.d16, sizeof(uint16_t) * slots));
            MLEM_CUDA(cudaMalloc(&op.dval, val_bytes(op.vt) * slots));
        }
        if (fits && op.nrows) {
            switch (op.vt) {
                case MLEM_VAL_F32: d16_fill<float>(op, idx, val, s); break;
                case MLEM_VAL_F16: d16_fill<__half>(op, idx, val, s); break;
                default: d16_fill<__nv_bfloat16>(op, idx, val, s);
            }
        }
        MLEM_CUDA(cudaStreamSynchronize(s));
    } catch (...) {
        cudaStreamSynchronize(s);
        cudaFree(word);
        cudaFree(nvec);
        cudaFree(sidx);
        cudaFree(sval);
        free_d16(op);
        throw;
    }
    cudaFree(word);
    cudaFree(nvec);
    cudaFree(sidx);
    cudaFree(sval);
    if (!fits) free_d16(op);
    return fits;
}

void launch_csr_d16(const DevCsr& op, const float* x, const EpiArgs& epi, int unroll, L2Window win, cudaStream_t s) {
    if (op.nrows) d16_dispatch(op, {}, x, epi, unroll, win, s);
}

void launch_merge_d16(const DevCsr& op, const MergePlan& p, const float* x, const EpiArgs& epi, int unroll,
                      L2Window win, cudaStream_t s) {
    if (p.ntiles) d16_dispatch(op, {p.tile_i, p.ntiles}, x, epi, unroll, win, s);
}

}  // namespace mlem
