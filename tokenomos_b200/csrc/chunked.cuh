// A recurrence with a state S [V, N] per head and a decay per head and token,
//
//     S_t = a_t S_(t-1) + w_t x_t b_t^T        y_t = S_t c_t (+ D x_t)         (x: V, b and c: N)
//
// is linear in S, so a portion of many tokens need not be walked one by one: over a chunk of CH_T tokens it is three matrix
// products, all chunks side by side but for one pass that carries the states along. With A_t the product of the chunk's
// decays up to t and S_0 the state before it,
//
//     gram:   G = c b^T                                                      per chunk and group of heads that share b and c
//     add:    dS = sum_t (A_end / A_t) w_t x_t b_t^T                         per chunk and head
//     carry:  S_0 <- A_end S_0 + dS, every chunk's S_0 left in dS's place    along the chunks
//     out:    y_t = A_t S_0 c_t + sum_{s <= t} (A_t / A_s) w_s G[t, s] x_s   per chunk and head
//
// Everything is 32-bit multiply-adds; the logarithms of the decays are summed, and subtracted, in 64-bit, so that a quotient
// of decays is as exact as the product of its factors. A walk has one chain of dependent steps per token and a few warps an
// SM to hide it behind (340 cycles a token); the products fill the GPU and read shared memory 16 bytes for 16 multiply-adds.
// A thread of 256 holds 4 x 4 outputs as pairs over two halves of the inner dimension (packed multiply-adds), both operands
// as rows along it.
//
// Chunks count from each sequence's first token of the step. Sequence s has the slots cu_seqlens[s] / CH_T + s and up, so that
// all sequences together need at most tokens / CH_T + n_seqs of them, whatever their lengths (a captured step does not know
// them); slots without tokens return at once, and so do warps whose rows lie behind a short chunk's end.
#pragma once

#include <math.h>

#include "packed.cuh"

namespace {

constexpr int CH_T = 64, CH_V = 64, CH_LD = CH_T + 4, CH_THREADS = 256, CH_MAX_N = 128;

struct ChunkRows {                 // rows of one operand: element (group, token, i) at base[group * group_stride + token * stride + i]
    const void* base;
    int64_t group_stride, stride;
};

struct Chunked {
    ChunkRows x, b, c;
    const int *cu_seqlens, *seq_ctx, *seq_slot;
    int n_seqs, H, V, N, groups;   // groups: heads / groups heads share b and c
    float* gram;                   // [slots][groups][CH_T][CH_T]
    float* carry;                  // [slots][H][V][N]
    float* chunk_decay;            // [slots][H]
    float* y;                      // [T, H V]
    float* state;                  // [request slots][H][N][V]
    int check;                     // the kernel's number in the index checks
};

// The decays of the state-space mixer: log a = -exp(A_log) dt, w = dt = softplus(dt_raw + bias), D x joins the output
struct SsdDecay {
    const float* dt_raw;
    int64_t dt_stride;
    const float *bias, *A_log, *D_skip;
    __device__ __forceinline__ void at(int token, int h, double& log_a, float& w) const {
        const float v = dt_raw[(size_t)token * dt_stride + h] + bias[h];
        const float dt = v > 20.f ? v : log1pf(expf(v));
        // (a decay of 0 keeps a finite logarithm: differences of two infinite ones would be NaN)
        const double la = -(double)expf(A_log[h]) * (double)dt;
        log_a = la < -1e6 ? -1e6 : la;
        w = dt;
    }
    __device__ __forceinline__ float skip(int h) const { return D_skip[h]; }
};

__device__ __forceinline__ void ch_zero(float2 (&acc)[4][4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = make_float2(0.f, 0.f);
}

struct ChunkAt {
    int s, j, first, nt;           // sequence, its chunk, the chunk's first token in the step and its count (0: no such chunk)
};
__device__ __forceinline__ ChunkAt chunk_at(const Chunked& m, int slot) {
    // the last sequence whose first slot is not past this one (every warp looks for itself, 32 sequences at a time)
    int lo = -1;
    for (int s0 = 0; s0 < m.n_seqs; s0 += 32) {
        const int s = s0 + (threadIdx.x & 31);
        const unsigned before = __ballot_sync(0xffffffffu, s < m.n_seqs && m.cu_seqlens[s] / CH_T + s <= slot);
        lo += __popc(before);
        if (before != 0xffffffffu) break;
    }
    ChunkAt c;
    c.s = lo;
    const int first = m.cu_seqlens[lo], len = m.cu_seqlens[lo + 1] - first;
    c.j = slot - (first / CH_T + lo);
    c.first = first + c.j * CH_T;
    c.nt = max(0, min(CH_T, len - c.j * CH_T));
    return c;
}

// cum[t]: log of the decays up to and with token t of the chunk; w[t] (0 past the end, where cum stays). By warps 0 and 1.
__device__ __forceinline__ void chunk_decays(const SsdDecay& d, const ChunkAt& c, int h, double* cum, float* w) {
    __shared__ double half_s;
    const int t = threadIdx.x, lane = t & 31;
    double la = 0.0;
    float wt = 0.f;
    if (t < CH_T && t < c.nt) d.at(c.first + t, h, la, wt);
    if (t < CH_T) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double up = __shfl_up_sync(0xffffffffu, la, o);
            if (lane >= o) la += up;
        }
        if (t == 31) half_s = la;
        w[t] = wt;
    }
    __syncthreads();
    if (t < CH_T) cum[t] = t >= 32 ? la + half_s : la;
    __syncthreads();
}

// Rows of an operand into shared memory as they are ([token][i], ld floats apart), zeros past the chunk's end
template <typename T>
__device__ __forceinline__ void chunk_rows(const ChunkRows& r, int group, const ChunkAt& c, int n, float* dst, int ld) {
    const T* base = (const T*)r.base + (size_t)group * r.group_stride;
    for (int i = threadIdx.x; i < CH_T * (n / 4); i += CH_THREADS) {
        const int t = i / (n / 4), k = i % (n / 4) * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t < c.nt) v = Quad<T>::load(base + (size_t)(c.first + t) * r.stride + k);
        *reinterpret_cast<float4*>(dst + t * ld + k) = v;
    }
}
// The same turned round ([i][token], CH_LD apart), each token's elements times scale[token] (null: as they are)
template <typename T>
__device__ __forceinline__ void chunk_turned(const ChunkRows& r, int group, const ChunkAt& c, int first, int n, const float* scale,
                                             float* dst) {
    const T* base = (const T*)r.base + (size_t)group * r.group_stride + first;
    for (int i = threadIdx.x; i < CH_T * (n / 4); i += CH_THREADS) {
        const int t = i % CH_T, k = i / CH_T * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t < c.nt) v = Quad<T>::load(base + (size_t)(c.first + t) * r.stride + k);
        const float f = scale != nullptr ? scale[t] : 1.f;
        dst[k * CH_LD + t] = v.x * f;
        dst[(k + 1) * CH_LD + t] = v.y * f;
        dst[(k + 2) * CH_LD + t] = v.z * f;
        dst[(k + 3) * CH_LD + t] = v.w * f;
    }
}

template <typename T>
__global__ void __launch_bounds__(CH_THREADS, 2) chunk_gram_kernel(const Chunked m) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float smem[];
    const int slot = blockIdx.x, g = blockIdx.y, tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const ChunkAt c = chunk_at(m, slot);
    if (c.nt == 0) return;
    const int ld = m.N + 4;
    float *Cs = smem, *Bs = smem + CH_T * ld;
    chunk_rows<T>(m.c, g, c, m.N, Cs, ld);
    chunk_rows<T>(m.b, g, c, m.N, Bs, ld);
    __syncthreads();
    if ((ty & ~1) * 4 >= c.nt) return;
    float2 acc[4][4];
    ch_zero(acc);
    tile_product<2>(Cs + ty * 4 * ld, ld, Bs + tx * ld, ld, m.N, acc);
    float* out = m.gram + ((size_t)slot * m.groups + g) * CH_T * CH_T;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) out[(ty * 4 + i) * CH_T + tx + 16 * j] = acc[i][j].x + acc[i][j].y;
}

template <typename T>
__global__ void __launch_bounds__(CH_THREADS, 2) chunk_add_kernel(const Chunked m, const SsdDecay d) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float smem[];
    __shared__ double cum[CH_T];
    __shared__ float w[CH_T];
    const int slot = blockIdx.x, h = blockIdx.y, v0 = blockIdx.z * CH_V, tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const ChunkAt c = chunk_at(m, slot);
    if (c.nt == 0) return;
    float *Xt = smem, *Bt = smem + CH_V * CH_LD;
    chunk_decays(d, c, h, cum, w);
    if (threadIdx.x < CH_T) w[threadIdx.x] *= expf((float)(cum[CH_T - 1] - cum[threadIdx.x]));
    if (threadIdx.x == 0 && v0 == 0) m.chunk_decay[(size_t)slot * m.H + h] = expf((float)cum[CH_T - 1]);
    __syncthreads();
    chunk_turned<T>(m.x, h, c, v0, CH_V, w, Xt);
    chunk_turned<T>(m.b, h / (m.H / m.groups), c, 0, m.N, nullptr, Bt);
    __syncthreads();
    const int K = (c.nt + 3) & ~3;
    for (int n0 = 0; n0 < m.N; n0 += 64) {
        float2 acc[4][4];
        ch_zero(acc);
        tile_product<2>(Xt + ty * 4 * CH_LD, CH_LD, Bt + (n0 + tx) * CH_LD, CH_LD, K, acc);
        float* out = m.carry + (((size_t)slot * m.H + h) * m.V + v0 + ty * 4) * m.N + n0 + tx;
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) out[(size_t)i * m.N + 16 * j] = acc[i][j].x + acc[i][j].y;
    }
}

// A thread carries four neighbouring elements (of N) of one state along its sequence's chunks, several chunks' loads in flight
__global__ void __launch_bounds__(128) chunk_carry_kernel(const Chunked m) {
    pdl_launch_dependents();
    pdl_wait();
    constexpr int AHEAD = 8;
    const int s = blockIdx.y, first = m.cu_seqlens[s], len = m.cu_seqlens[s + 1] - first;
    const int64_t cells = (int64_t)m.H * m.V * m.N, e = ((int64_t)blockIdx.x * 128 + threadIdx.x) * 4;
    if (len <= 0 || e >= cells) return;
    const int n_chunks = (len + CH_T - 1) / CH_T, slot0 = first / CH_T + s;
    const int h = (int)(e / ((int64_t)m.V * m.N)), v = (int)(e / m.N % m.V), n = (int)(e % m.N);
    float* st = m.state + (size_t)TK_SLOT(m.check, m.seq_slot[s]) * cells + (size_t)h * m.V * m.N;
    const int64_t at = (int64_t)n * m.V + v, step = m.V;
    float4 S = make_float4(0.f, 0.f, 0.f, 0.f);
    if (m.seq_ctx[s] > 0) S = make_float4(st[at], st[at + step], st[at + 2 * step], st[at + 3 * step]);
    float* cell = m.carry + (size_t)slot0 * cells + e;
    const float* dec = m.chunk_decay + (size_t)slot0 * m.H + h;
    for (int j0 = 0; j0 < n_chunks; j0 += AHEAD) {
        float4 add[AHEAD];
        float a[AHEAD];
#pragma unroll
        for (int i = 0; i < AHEAD; ++i)
            if (j0 + i < n_chunks) {
                add[i] = *reinterpret_cast<const float4*>(cell + (size_t)(j0 + i) * cells);
                a[i] = dec[(size_t)(j0 + i) * m.H];
            }
#pragma unroll
        for (int i = 0; i < AHEAD; ++i)
            if (j0 + i < n_chunks) {
                *reinterpret_cast<float4*>(cell + (size_t)(j0 + i) * cells) = S;
                S.x = fmaf(a[i], S.x, add[i].x);
                S.y = fmaf(a[i], S.y, add[i].y);
                S.z = fmaf(a[i], S.z, add[i].z);
                S.w = fmaf(a[i], S.w, add[i].w);
            }
    }
    st[at] = S.x;
    st[at + step] = S.y;
    st[at + 2 * step] = S.z;
    st[at + 3 * step] = S.w;
}

template <typename T>
__global__ void __launch_bounds__(CH_THREADS, 2) chunk_out_kernel(const Chunked m, const SsdDecay d) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float smem[];
    __shared__ double cum[CH_T];
    __shared__ float w[CH_T];
    const int slot = blockIdx.x, h = blockIdx.y, v0 = blockIdx.z * CH_V, tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const ChunkAt c = chunk_at(m, slot);
    if (c.nt == 0) return;
    const int ld = m.N + 4, g = h / (m.H / m.groups);
    float *Cs = smem, *St = Cs + CH_T * ld, *Ms = St + CH_V * ld, *Xt = Ms + CH_T * CH_LD;
    const bool fresh = c.j == 0 && m.seq_ctx[c.s] == 0;           // nothing came before
    chunk_decays(d, c, h, cum, w);
    if (!fresh) {
        chunk_rows<T>(m.c, g, c, m.N, Cs, ld);
        const float* S0 = m.carry + (((size_t)slot * m.H + h) * m.V + v0) * m.N;
        for (int i = tid; i < CH_V * (m.N / 4); i += CH_THREADS)
            *reinterpret_cast<float4*>(St + i / (m.N / 4) * ld + i % (m.N / 4) * 4) = *reinterpret_cast<const float4*>(S0 + 4 * i);
    }
    chunk_turned<T>(m.x, h, c, v0, CH_V, nullptr, Xt);
    const float* gram = m.gram + ((size_t)slot * m.groups + g) * CH_T * CH_T;
    for (int i = tid; i < CH_T * CH_T; i += CH_THREADS) {
        const int t = i / CH_T, s = i % CH_T;
        Ms[t * CH_LD + s] = s <= t && t < c.nt ? gram[i] * (expf((float)(cum[t] - cum[s])) * w[s]) : 0.f;
    }
    __syncthreads();
    const int row0 = (ty & ~1) * 4;                               // the warp's first row
    if (row0 >= c.nt) return;
    float2 acc[4][4];
    ch_zero(acc);
    if (!fresh) {
        tile_product<2>(Cs + ty * 4 * ld, ld, St + tx * ld, ld, m.N, acc);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float a = expf((float)cum[ty * 4 + i]);
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j].x *= a, acc[i][j].y *= a;
        }
    }
    tile_product<2>(Ms + ty * 4 * CH_LD, CH_LD, Xt + tx * CH_LD, CH_LD, row0, acc);
    // the warp's own eight columns, where a row ends: what comes after a token stays out of its sum, whatever it holds
#pragma unroll
    for (int s = 0; s < 8; ++s) {
        float xv[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) xv[j] = Xt[(tx + 16 * j) * CH_LD + row0 + s];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (row0 + s > ty * 4 + i) continue;
            const float wt = Ms[(ty * 4 + i) * CH_LD + row0 + s];
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j].x = fmaf(wt, xv[j], acc[i][j].x);
        }
    }
    const float D = d.skip(h);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int t = ty * 4 + i;
        if (t >= c.nt) continue;
        float* out = m.y + (size_t)(c.first + t) * m.H * m.V + h * m.V + v0 + tx;
#pragma unroll
        for (int j = 0; j < 4; ++j) out[16 * j] = fmaf(D, Xt[(tx + 16 * j) * CH_LD + t], acc[i][j].x + acc[i][j].y);
    }
}

// What the four kernels take: whole 16-byte pieces, blocks of 64 rows of the state, its columns in one or two halves of 64.
inline bool chunked_takes(int V, int N) { return V > 0 && V % CH_V == 0 && (N == 64 || N == CH_MAX_N); }

// float32 words of scratch for a step of `tokens` tokens in `n_seqs` sequences: gram, carry, chunk_decay in that order
inline int64_t chunked_scratch(int64_t tokens, int64_t n_seqs, int64_t H, int64_t V, int64_t N, int64_t groups) {
    const int64_t slots = tokens / CH_T + n_seqs;
    return slots * (groups * CH_T * CH_T + H * V * N + (H + 3) / 4 * 4);
}

template <typename T>
int launch_chunked(Chunked m, const SsdDecay& d, float* scratch, int tokens, cudaStream_t stream) {
    const int slots = tokens / CH_T + m.n_seqs, ld = m.N + 4, vb = m.V / CH_V;
    m.gram = scratch;
    m.carry = m.gram + (size_t)slots * m.groups * CH_T * CH_T;
    m.chunk_decay = m.carry + (size_t)slots * m.H * m.V * m.N;
    const int gram_smem = 2 * CH_T * ld * 4, add_smem = (CH_V + m.N) * CH_LD * 4;
    const int out_smem = ((CH_T + CH_V) * ld + (CH_T + CH_V) * CH_LD) * 4;
    cudaFuncSetAttribute(chunk_gram_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, gram_smem);
    cudaFuncSetAttribute(chunk_add_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, add_smem);
    cudaFuncSetAttribute(chunk_out_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, out_smem);
    tk_launch(chunk_gram_kernel<T>, dim3(slots, m.groups), dim3(CH_THREADS), gram_smem, stream, m);
    TK_CHECK_LAUNCH("chunk_gram");
    tk_launch(chunk_add_kernel<T>, dim3(slots, m.H, vb), dim3(CH_THREADS), add_smem, stream, m, d);
    TK_CHECK_LAUNCH("chunk_add");
    const int64_t quads = (int64_t)m.H * m.V * m.N / 4;
    tk_launch(chunk_carry_kernel, dim3((unsigned)((quads + 127) / 128), m.n_seqs), dim3(128), 0, stream, m);
    TK_CHECK_LAUNCH("chunk_carry");
    tk_launch(chunk_out_kernel<T>, dim3(slots, m.H, vb), dim3(CH_THREADS), out_smem, stream, m, d);
    TK_CHECK_LAUNCH("chunk_out");
    return 0;
}

}  // namespace
