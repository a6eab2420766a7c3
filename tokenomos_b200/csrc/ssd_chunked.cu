// The state-space recurrence (ssd.cu) chunk by chunk on the tensor cores, for 16-bit x, B and C:
//
//     S_t = a_t S_(t-1) + w_t x_t b_t^T        y_t = S_t c_t + D x_t        (S: V x N per head, 32-bit; w = dt, a = exp(-A dt))
//
// Over a chunk of 64 tokens, A_t the product of its decays up to t and S_0 the state before it,
//
//     Y = diag(A) C S_0^T + M X + D X        S_0 <- A_end S_0 + X^T diag(w A_end / A) B        M[t, s] = (A_t / A_s) w_s c_t . b_s
//
// The first kernel forms M of all chunks side by side, the second walks each head's chunks with S in the accumulators of mma.sync;
// arithmetic, layout and what becomes of numbers that are not finite are those of delta_chunked.cu: x, b and c are 16-bit
// numbers as they are, the floats beside them (S, M, the weighted x) come in three 16-bit parts, so products are exact up to the
// sums.
//
// Four warps own 16 rows of V: two carry S (half of N's columns each), whose parts they hand on, and add a chunk to it, two write
// the chunk's outputs (half of the tokens each); one barrier a chunk. What bounds it is the longer of the two chains, 1,800
// cycles a chunk of 64 x 128 (96 products of 8 cycles in one, 126 in the other, and taking floats apart). Measured (both kernels; in
// brackets multiply-adds over chunks, and the walk): 32 heads of 64 x 128 on 2,048 tokens 63 us (144, 368), 64 heads 92 (274, 496),
// eight sequences of 512 164 (-, 495), one of 64 12 (-, 20). Against 64 bits y is 6e-8 to 8e-8 off and S 1e-7, the walk 6e-8 to 3e-7
// and 1e-7 to 7e-7.
#include "chunk_tc.cuh"

namespace {
enum : int { TK_K_SSD_CHUNKS = 17 };
// factors of a chunk's tokens (one array of 64 each): A_t; w_t A_end / A_t; A_end (first element)
enum : int { SC_A = 0, SC_W = 1, SC_END = 2, SC_FACTORS = 3 };
constexpr int SC_MAT = 3 * DC_PART;            // bytes of a chunk's and head's M
constexpr int64_t SC_WORDS = SC_MAT / 4 + SC_FACTORS * DC_T;       // floats of scratch a chunk and head

struct SsdChunks {
    const __nv_bfloat16 *x, *b, *c;            // rows `stride` apart: x [H][V], b and c [G][N]
    int64_t stride;
    const float* dt_raw;
    int64_t dt_stride;
    const float *bias, *A_log, *D_skip;
    float* state;                              // [request slots][H][N][V]
    const int *cu_seqlens, *seq_ctx, *seq_slot;
    int n_seqs;
    float* y;
    int H, G, V;
    uint8_t* mats;                             // [slots][H][three parts]
    float* factors;                            // [slots][H][SC_FACTORS][64]
};

// M of one chunk and two heads of a group, four warps each.
template <int N>
__global__ void __launch_bounds__(256, 3)
ssd_chunk_prepare_kernel(const SsdChunks m) {
    extern __shared__ __align__(128) uint8_t prep_smem[];
    constexpr int TILE = DC_T * N * 2;
    float* gram = reinterpret_cast<float*>(prep_smem + 2 * TILE);
    __shared__ double half_s[2];
    __shared__ float2 cum_s[2][DC_T];          // the logarithms' sums as two floats: their differences are as exact as 64-bit ones
    __shared__ __align__(8) float w_s[2][DC_T];
    pdl_launch_dependents();
    pdl_wait();
    const int per = m.H / m.G, pairs = (per + 1) / 2, slot = blockIdx.x, g = blockIdx.y / pairs;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, which = warp >> 2, quarter = warp & 3, t = tid & 63;
    const Chunk64 at = chunk_of(m.cu_seqlens, m.n_seqs, slot);
    const int first = at.first, nt = at.nt;
    if (nt <= 0) return;
    const uint32_t bt = shared_u32(prep_smem), ct = bt + TILE;
#pragma unroll
    for (int i = tid; i < DC_T * (N / 8); i += 256) {
        const int r = i / (N / 8), k = i % (N / 8);
        const int64_t off = (int64_t)(first + (r < nt ? r : 0)) * m.stride + g * N + k * 8;
        cp_async16(bt + tile_off<N>(r, k), m.b + off, r < nt);
        cp_async16(ct + tile_off<N>(r, k), m.c + off, r < nt);
    }
    cp_async_commit();
    // meanwhile the decays
    const int in_group = blockIdx.y % pairs * 2 + which, h = g * per + in_group;
    const bool live = in_group < per;
    double la = 0.0;
    float w = 0.f;
    if (quarter < 2) {
        if (live && t < nt) {
            const float v = m.dt_raw[(size_t)(first + t) * m.dt_stride + h] + m.bias[h];
            w = v > 20.f ? v : log1pf(expf(v));
            // (a decay of 0 keeps a finite logarithm: differences of two infinite ones would be NaN)
            la = -(double)expf(m.A_log[h]) * (double)w;
            la = la < -1e6 ? -1e6 : la;
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double up = __shfl_up_sync(0xffffffffu, la, o);
            if (lane >= o) la += up;
        }
        if (t == 31) half_s[which] = la;
    }
    cp_async_wait<0>();
    __syncthreads();
    for (int n = warp; n < 10; n += 8) lower_block<N>(gram, ct, bt, n, lane);
    if (quarter < 2) {
        if (t >= 32) la += half_s[which];
        cum_s[which][t] = make_float2((float)la, (float)(la - (double)(float)la));
        w_s[which][t] = w;
    }
    __syncthreads();
    if (!live) return;
    if (quarter < 2) {
        const float2 last = cum_s[which][DC_T - 1];
        const double end = (double)last.x + (double)last.y;
        float* f = m.factors + ((size_t)slot * m.H + h) * SC_FACTORS * DC_T;
        f[SC_A * DC_T + t] = expf((float)la);
        f[SC_W * DC_T + t] = w * expf((float)(end - la));
        if (t == 0) f[SC_END * DC_T] = expf((float)end);
    }
    uint8_t* mat = m.mats + ((size_t)slot * m.H + h) * SC_MAT;
#pragma unroll
    for (int n = 0; n < DC_STEPS; ++n) {
        const int2 p = triangle_step(n, quarter, lane);
        const int k = p.y & (DC_T - 2);
        const float2 ri = cum_s[which][p.x], a0 = cum_s[which][k], a1 = cum_s[which][k + 1];
        const float2 wk = *reinterpret_cast<const float2*>(&w_s[which][k]);
        const float2 cb = *reinterpret_cast<const float2*>(gram + p.x * DC_LD + k);
        const float v0 = cb.x * (expf((ri.x - a0.x) + (ri.y - a0.y)) * wk.x);
        const float v1 = cb.y * (expf((ri.x - a1.x) + (ri.y - a1.y)) * wk.y);
        if (p.y >= DC_T) continue;
        store_parts(mat, p, k <= p.x ? v0 : 0.f, k < p.x ? v1 : 0.f);
    }
}

template <int N, int PAIRS>
struct ScSmem {
    static constexpr int TILE = DC_T * N * 2, XROW = PAIRS * 32 + 16;
    static constexpr int B = 0, C = B + TILE, M = C + TILE, X = M + SC_MAT, F = X + DC_T * XROW, STAGE = F + SC_FACTORS * DC_T * 4;
    static constexpr int S = 2 * STAGE, S_BYTES = PAIRS * (N / 16) * 3 * 512, ALL = S + 2 * S_BYTES;
};

template <int N, int PAIRS>
__global__ void __launch_bounds__(128 * PAIRS, 1)
ssd_chunk_walk_kernel(const SsdChunks m) {
    using Z = ScSmem<N, PAIRS>;
    constexpr int THREADS = 128 * PAIRS, NH = N / 2, KS = NH / 16, NS = NH / 8, COLS = 16 * PAIRS;
    extern __shared__ __align__(128) uint8_t walk_smem[];
    const uint32_t base = shared_u32(walk_smem);
    pdl_launch_dependents();
    pdl_wait();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, pair = (warp % (2 * PAIRS)) >> 1, half = warp & 1;
    const int c0 = blockIdx.x * COLS, h = blockIdx.y, s = blockIdx.z, g = h / (m.H / m.G);
    const int begin = m.cu_seqlens[s], len = m.cu_seqlens[s + 1] - begin;
    if (len <= 0) return;
    const int n_chunks = (len + DC_T - 1) / DC_T, slot0 = begin / DC_T + s;
    const int row = lane >> 2, tok = 2 * (lane & 3);            // the accumulators' row (and row + 8) and first column of eight
    const int v0 = c0 + pair * 16 + row;
    const uint32_t b_row = (lane & 7) + (lane >> 4) * 8, b_chunk = (lane >> 3) & 1;      // ldmatrix rows of a right operand
    auto load = [&](int j) {
        if (j < n_chunks) {
            const uint32_t to = base + (j & 1) * Z::STAGE;
            const int first = begin + j * DC_T, nt = len - j * DC_T;
#pragma unroll
            for (int i = tid; i < DC_T * (N / 8); i += THREADS) {
                const int r = i / (N / 8), k = i % (N / 8);
                const int64_t off = (int64_t)(first + (r < nt ? r : 0)) * m.stride + g * N + k * 8;
                cp_async16(to + Z::B + tile_off<N>(r, k), m.b + off, r < nt);
                cp_async16(to + Z::C + tile_off<N>(r, k), m.c + off, r < nt);
            }
            const uint8_t* mat = m.mats + ((size_t)(slot0 + j) * m.H + h) * SC_MAT;
#pragma unroll
            for (int i = tid; i < SC_MAT / 16; i += THREADS) cp_async16(to + Z::M + i * 16, mat + i * 16, true);
#pragma unroll
            for (int i = tid; i < DC_T * (COLS / 8); i += THREADS) {
                const int r = i / (COLS / 8), k = i % (COLS / 8);
                cp_async16(to + Z::X + r * Z::XROW + k * 16,
                           m.x + (int64_t)(first + (r < nt ? r : 0)) * m.stride + h * m.V + c0 + k * 8, r < nt);
            }
            const float* f = m.factors + ((size_t)(slot0 + j) * m.H + h) * SC_FACTORS * DC_T;
            for (int i = tid; i < SC_FACTORS * DC_T / 4; i += THREADS) cp_async16(to + Z::F + i * 16, f + i * 4, true);
        }
        cp_async_commit();
    };
    uint8_t* const s_parts = walk_smem + Z::S + pair * (N / 16) * 3 * 512 + lane * 16;
    load(0);

    if (warp < 2 * PAIRS) {
        float* st = m.state + ((size_t)TK_SLOT(TK_K_SSD_CHUNKS, m.seq_slot[s]) * m.H + h) * N * m.V + (size_t)(half * NH + tok) * m.V + v0;
        float S[NS][4];
        const bool carried = m.seq_ctx[s] > 0;
#pragma unroll
        for (int n = 0; n < NS; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) S[n][e] = carried ? st[(size_t)(n * 8 + (e & 1)) * m.V + (e >> 1) * 8] : 0.f;
        for (int j = 0; j < n_chunks; ++j) {
            const uint32_t at = base + (j & 1) * Z::STAGE;
            const float* f = reinterpret_cast<const float*>(walk_smem + (j & 1) * Z::STAGE + Z::F);
#pragma unroll
            for (int ks = 0; ks < KS; ++ks) {
                uint32_t a[3][4];
                dc_cut(a, S[2 * ks], S[2 * ks + 1]);
                dc_give(s_parts + (j & 1) * Z::S_BYTES + (half * KS + ks) * 3 * 512, a);
            }
            cp_async_wait<0>();
            dc_sync();                                          // the chunk and S's parts are there, the chunk before is read
            load(j + 1);
            float hi[NS][4], hi2[NS][4], lo[NS][4];             // (high parts in two chains: half the sums that are cut off)
            dc_zero(hi);
            dc_zero(hi2);
            dc_zero(lo);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                uint32_t xx[4], a[3][4], b[NS / 2][4];          // x: (8 tokens, rows 0-7), (rows 8-15), the next 8 tokens
                ldmatrix_x4_trans(xx, at + Z::X + (k * 16 + b_row) * Z::XROW + pair * 32 + b_chunk * 16);
#pragma unroll
                for (int np = 0; np < NS / 2; ++np)
                    ldmatrix_x4_trans(b[np], at + Z::B + tile_off<N>(k * 16 + (lane & 15), half * (NH / 8) + np * 2 + (lane >> 4)));
                float u[2][4];
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const float2 w = *reinterpret_cast<const float2*>(f + SC_W * DC_T + (2 * k + q) * 8 + tok);
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        u[q][2 * r] = __uint_as_float(xx[2 * q + r] << 16) * w.x;
                        u[q][2 * r + 1] = __uint_as_float(xx[2 * q + r] & 0xffff0000u) * w.y;
                    }
                }
                dc_cut(a, u[0], u[1]);
                float(&top)[NS][4] = k & 1 ? hi2 : hi;
#pragma unroll
                for (int np = 0; np < NS / 2; ++np) dc_three(top[2 * np], top[2 * np + 1], lo[2 * np], lo[2 * np + 1], a, b[np]);
            }
            const float end = f[SC_END * DC_T];
#pragma unroll
            for (int n = 0; n < NS; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) S[n][e] = fmaf(end, S[n][e], hi[n][e] + hi2[n][e] + lo[n][e]);
        }
#pragma unroll
        for (int n = 0; n < NS; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) st[(size_t)(n * 8 + (e & 1)) * m.V + (e >> 1) * 8] = S[n][e];
        return;
    }

    const int HV = m.H * m.V;
    float* y = m.y + (size_t)begin * HV + h * m.V + v0;
    const float nan = __int_as_float(0x7fffffff), D = m.D_skip[h];
    // the tokens of this warp: blocks of 16 tokens 0 and 3, or 1 and 2 (the same number of blocks left of the diagonal)
    for (int j = 0; j < n_chunks; ++j) {
        const uint32_t at = base + (j & 1) * Z::STAGE;
        const float* f = reinterpret_cast<const float*>(walk_smem + (j & 1) * Z::STAGE + Z::F);
        cp_async_wait<0>();
        dc_sync();
        load(j + 1);
        float out[4][4];
        {
            float hi[4][4], hi2[4][4], lo[4][4];
            dc_zero(hi);
            dc_zero(hi2);
            dc_zero(lo);
#pragma unroll
            for (int ks = 0; ks < N / 16; ++ks) {
                uint32_t a[3][4], b[4], b2[4];
                dc_take(a, s_parts + (j & 1) * Z::S_BYTES + ks * 3 * 512);
                ldmatrix_x4(b, at + Z::C + tile_off<N>(half * 16 + b_row, ks * 2 + b_chunk));
                ldmatrix_x4(b2, at + Z::C + tile_off<N>((3 - half) * 16 + b_row, ks * 2 + b_chunk));
                float(&top)[4][4] = ks & 1 ? hi2 : hi;
                dc_three(top[0], top[1], lo[0], lo[1], a, b);
                dc_three(top[2], top[3], lo[2], lo[3], a, b2);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float2 w = *reinterpret_cast<const float2*>(f + SC_A * DC_T + (i < 2 ? half : 3 - half) * 16 + (i & 1) * 8 + tok);
#pragma unroll
                for (int e = 0; e < 4; ++e) out[i][e] = (e & 1 ? w.y : w.x) * (hi[i][e] + hi2[i][e] + lo[i][e]);
            }
        }
        float hi[4][4], hi2[4][4], lo[4][4];
        dc_zero(hi);
        dc_zero(hi2);
        dc_zero(lo);
        int odd0 = DC_T, odd1 = DC_T;                           // the first token of rows row and row + 8 that is not finite
        uint32_t own[2][4];                                     // x of this warp's tokens, as the accumulators hold them
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (k > 3 - half) continue;
            uint32_t xx[4];                                     // x, turned round: a left operand as it is
            ldmatrix_x4_trans(xx, at + Z::X + (k * 16 + b_row) * Z::XROW + pair * 32 + b_chunk * 16);
            bool odd = false;
#pragma unroll
            for (int e = 0; e < 4; ++e) odd = odd || (xx[e] & 0x7f80u) == 0x7f80u || (xx[e] & 0x7f800000u) == 0x7f800000u;
            if (__any_sync(0xffffffffu, odd)) {
#pragma unroll
                for (int e = 0; e < 8; ++e) {                   // (register e >> 1: rows row, row + 8 by its first bit, tokens 8 further by its second)
                    const uint32_t mask = e & 1 ? 0x7f800000u : 0x7f80u;
                    if ((xx[e >> 1] & mask) != mask) continue;
                    xx[e >> 1] &= e & 1 ? 0xffffu : 0xffff0000u;
                    int& first = (e >> 1) & 1 ? odd1 : odd0;
                    first = min(first, k * 16 + (e >> 2) * 8 + tok + (e & 1));
                }
            }
#pragma unroll
            for (int i = 0; i < 2; ++i) {                       // the later block of tokens first: the earlier one may lie before k
                const int block = i ? half : 3 - half, q = i ? 0 : 2;
                if (k > block) continue;
                if (k == block) own[1 - i][0] = xx[0], own[1 - i][1] = xx[1], own[1 - i][2] = xx[2], own[1 - i][3] = xx[3];
                const uint32_t mt = at + Z::M + tile_off<DC_T>(block * 16 + b_row, k * 2 + b_chunk);
                uint32_t b[3][4];
#pragma unroll
                for (int p = 0; p < 3; ++p) ldmatrix_x4(b[p], mt + p * DC_PART);
                mma16816(lo[q], xx, b[2][0], b[2][1]);
                mma16816(lo[q + 1], xx, b[2][2], b[2][3]);
                float(&top)[4][4] = k & 1 ? hi2 : hi;
                mma16816(top[q], xx, b[0][0], b[0][1]);
                mma16816(top[q + 1], xx, b[0][2], b[0][3]);
                mma16816(lo[q], xx, b[1][0], b[1][1]);
                mma16816(lo[q + 1], xx, b[1][2], b[1][3]);
            }
        }
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) {
            odd0 = min(odd0, __shfl_xor_sync(0xffffffffu, odd0, o));
            odd1 = min(odd1, __shfl_xor_sync(0xffffffffu, odd1, o));
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int t = (i < 2 ? half : 3 - half) * 16 + (i & 1) * 8 + tok;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const uint32_t x = own[i >> 1][(i & 1) * 2 + (e >> 1)];
                out[i][e] = fmaf(D, __uint_as_float(e & 1 ? x & 0xffff0000u : x << 16), out[i][e] + (hi[i][e] + hi2[i][e] + lo[i][e]));
                if (t + (e & 1) >= (e < 2 ? odd0 : odd1)) out[i][e] = nan;
            }
            float* dst = y + (size_t)(j * DC_T + t) * HV;
            if (j * DC_T + t < len) dst[0] = out[i][0], dst[8] = out[i][2];
            if (j * DC_T + t + 1 < len) dst[HV] = out[i][1], dst[HV + 8] = out[i][3];
        }
    }
}

template <int N, int PAIRS>
void sc_walk(const SsdChunks& m, cudaStream_t stream) {
    constexpr int smem = ScSmem<N, PAIRS>::ALL;
    auto kernel = ssd_chunk_walk_kernel<N, PAIRS>;
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    tk_launch_after(kernel, dim3(m.V / (16 * PAIRS), m.H, m.n_seqs), dim3(128 * PAIRS), smem, stream, m);
}

template <int N>
void sc_launch(const SsdChunks& m, int slots, int sm_count, cudaStream_t stream) {
    constexpr int smem = 2 * DC_T * N * 2 + DC_T * DC_LD * 4;
    auto prepare = ssd_chunk_prepare_kernel<N>;
    cudaFuncSetAttribute(prepare, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    tk_launch(prepare, dim3(slots, m.G * ((m.H / m.G + 1) / 2)), dim3(256), smem, stream, m);
    // 32 rows of V a block, 16 while those blocks all find an SM of their own
    if ((int64_t)m.V / 16 * m.H * m.n_seqs <= sm_count) sc_walk<N, 1>(m, stream);
    else sc_walk<N, 2>(m, stream);
}
}  // namespace

// Words of scratch of a step chunk by chunk on the tensor cores, or 0: not taken. From 48 tokens a sequence on the chunks are faster
// than the walk at every number of heads and sequences (us, chunks against walk: 32 heads of 64 x 128, one sequence of 48
// tokens 8.8 and 12.5, four 15.3 and 17.2, sixteen 34.8 and 57.7; 64 heads of 64 x 64, four 17.8 and 21.6; on 32 tokens 15.0 and
// 12.9, 17.6 and 16.1).
TK_API int tk_ssd_tc_scratch(int tokens, int n_seqs, int H, int V, int N, int G) {
    if ((N != 64 && N != 128) || V <= 0 || V % 32 != 0 || H <= 0 || G <= 0 || H % G != 0 || n_seqs <= 0 || n_seqs > 65535 || H > 32767) return 0;
    if (tokens < 48 * (int64_t)n_seqs) return 0;
    const int64_t words = ((int64_t)tokens / DC_T + n_seqs) * H * SC_WORDS;
    return words * 4 <= (int64_t)512 << 20 ? (int)words : 0;
}

// tk_ssd_scan over bfloat16 rows, y one part; rows and bases whole 16-byte pieces. scratch: what tk_ssd_tc_scratch says.
TK_API int tk_ssd_tc(const void* xbc, int64_t xbc_stride, const float* dt_raw, int64_t dt_stride, const float* dt_bias,
                     const float* A_log, const float* D_skip, float* state, const int* cu_seqlens, const int* seq_ctx,
                     const int* seq_slot, int n_seqs, int tokens, float* y, int H, int V, int N, int G, float* scratch,
                     int sm_count, cudaStream_t stream) {
    TK_CHECK_ARG(tk_ssd_tc_scratch(tokens, n_seqs, H, V, N, G) > 0 && scratch != nullptr,
                 "state-space chunks: %d tokens of %d sequences, heads of %d x %d", tokens, n_seqs, N, V);
    TK_CHECK_ARG(xbc_stride % 8 == 0 && (((uintptr_t)xbc | (uintptr_t)scratch) & 15) == 0,
                 "state-space chunks: rows must be whole 16-byte pieces");
    const __nv_bfloat16* rows = (const __nv_bfloat16*)xbc;
    const int slots = tokens / DC_T + n_seqs;
    const SsdChunks m{rows, rows + (int64_t)H * V, rows + (int64_t)H * V + (int64_t)G * N, xbc_stride, dt_raw, dt_stride, dt_bias, A_log,
                      D_skip, state, cu_seqlens, seq_ctx, seq_slot, n_seqs, y, H, G, V, reinterpret_cast<uint8_t*>(scratch),
                      scratch + (size_t)slots * H * (SC_MAT / 4)};
    if (N == 64) sc_launch<64>(m, slots, sm_count, stream);
    else sc_launch<128>(m, slots, sm_count, stream);
    TK_CHECK_LAUNCH("ssd_tc");
    return 0;
}
