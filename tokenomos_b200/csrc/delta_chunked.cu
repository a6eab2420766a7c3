// The delta rule with a decay per head, chunk by chunk on the tensor cores (16-bit q, k and v, unit keys; the walk token by
// token and the other forms: linmem.cu):
//
//     S <- a_t S;  u_t = beta_t (v_t - S k_t);  S <- S + u_t k_t^T;  o_t = S q_t            (S: V x D per head, 32-bit)
//
// Over a chunk of 64 tokens, with A_t the product of the decays up to t and S_0 the state before it, all u together solve
//
//     (1 + L) U = diag(beta) (V - diag(A) K S_0^T),     L[t, s] = beta_t (A_t / A_s) k_t . k_s   for s < t
//
// so that with T = (1 + L)^-1 diag(beta), which needs nothing of the state, a chunk is five products in a row:
//
//     P = K S_0^T,  P' = Q S_0^T;   R = V - diag(A) P;   U = T R;   O = diag(A) P' + G U;   S_0 <- A_end S_0 + U^T diag(A_end / A) K
//
// with G[t, s] = (A_t / A_s) q_t . k_s for s <= t. The first kernel forms T and G of all chunks side by side, the second walks
// each head's chunks. 32-bit arithmetic on 16-bit tensor cores (mma.sync): k and q are 16-bit numbers as they are (their
// lengths are factors of the tokens), so a product of a float with them takes the float's three 16-bit parts and is exact up to
// the sums; products of two floats take the six largest of nine. Sums of the high parts and of the rest are kept apart, and what a chunk
// adds joins S in 32-bit registers, because the tensor cores cut sums off where the adder rounds. The logarithms of the decays
// are summed and subtracted in 64-bit.
//
// The walk's layout: everything lives transposed, V rows by tokens, so that a warp that owns 16 rows of V keeps S, R and U in
// its accumulators and each is, without leaving the registers, the left operand of the next product; K, Q, T and G are the
// right operands and come from shared memory by ldmatrix. What bounds it is the chain of one warp's products from chunk to chunk
// (8 cycles an mma.sync of 16 x 8 x 16), so two warps share 16 rows: each forms half of D's sums of P and P', half of the tokens of U and
// O, and half of D's columns of S, and they exchange partial sums twice a chunk through shared memory.
//
// A number that is not finite reaches its own row of V from its token on, as in the walk, and nothing before: such elements of
// R and U are taken out of the products and every output of the row from the first one on, and the row of S, are set to NaN.
// (Products with k come before its length is divided out: values and states beyond 2^128 / |k| overflow, and k of 2^64 and more in two
// tokens of a chunk.)
//
// Measured (both kernels, us; token by token in brackets): 16 heads of 128 x 128 over 8 on 750 and 2,250 tokens 138 (462), on 2,048
// 112 (324); heads of 64 x 64 88 (314) and 78 (280); 16 x 16 heads of 128, sixteen sequences of 512, 251 (614). Against 64 bits, on
// what projections and convolutions of random weights give (fourteen cases of 72 to 3,000 tokens), y is 1.4e-7 to 1.7e-7 off and S 1.1e-7 to
// 1.4e-7, the walk 1.7e-7 to 9.5e-7 and 1.8e-7 to 1.2e-6 (growing with the tokens). Keys that share a direction (0.9 to all of it, or with
// alternating signs): 1.8e-7 to 2.4e-7 where gates forget within some ten tokens (the walk 1.4e-7 to 2.9e-7), 4.0e-7 to 6.0e-7 where
// they hardly do (3.6e-7 to 1.9e-6). A chunk takes 4,800 cycles of
// a state warp (P 1,050, R 450, U 900, its parts 600, the update of S 1,200 with its sums), of which 2,000 are its 252 products.
#include "chunk_tc.cuh"

namespace {
enum : int { TK_K_DELTA_CHUNKS = 16 };
constexpr int DC_MATS = 6 * DC_PART;           // bytes of a chunk's and head's T and G: three parts each
// factors of a chunk's tokens (one array of 64 each): A_t |k_t|^-1; A_t scale |q_t|^-1; (A_end / A_t) |k_t|^-1; A_end (first element)
enum : int { DC_K = 0, DC_Q = 1, DC_W = 2, DC_END = 3, DC_FACTORS = 4 };
constexpr int64_t DC_WORDS = DC_MATS / 4 + DC_FACTORS * DC_T;      // floats of scratch a chunk and head

struct DeltaChunks {
    const __nv_bfloat16* qkv;
    int64_t stride;
    int q_off, k_off, v_off;
    const float* zb;
    int64_t zb_stride;
    const float* za;
    int64_t za_stride;
    const float *bias, *A;
    float* state;
    const int *cu_seqlens, *seq_ctx, *seq_slot;
    int n_seqs;
    float* y;
    int H, K, V;
    float q_scale;
    uint8_t* mats;             // [slots][H][T's parts, G's parts], each part as the walk's shared memory holds it
    float* factors;            // [slots][H][DC_FACTORS][64]
};

// The matrix at L (rows DC_LD apart): its lower left block of B x B becomes -T22 (L21 T11), T11 and T22 being the blocks above and
// beside it; thread (r, c) has COLS neighbouring elements of row r. T11 is zero above its diagonal; the block above T22 is used, and
// zero afterwards. Rows of T22 L21 T11 read nothing of later rows, so that a row that is not finite reaches none before it.
template <int B, int COLS>
__device__ __forceinline__ void join_blocks(float* L, int r, int c, bool live) {
    float *low = L + (B + r) * DC_LD, *temp = L + B + c;
    auto add = [&](float2 (&acc)[COLS / 2], float f, const float* src) {
#pragma unroll
        for (int i = 0; i < COLS / 2; i += 2) {
            const float4 v = *reinterpret_cast<const float4*>(src + 2 * i);
            acc[i] = fma2(make_float2(f, f), make_float2(v.x, v.y), acc[i]);
            acc[i + 1] = fma2(make_float2(f, f), make_float2(v.z, v.w), acc[i + 1]);
        }
    };
    float2 acc[COLS / 2];
#pragma unroll
    for (int i = 0; i < COLS / 2; ++i) acc[i] = make_float2(0.f, 0.f);
    if (live) {
#pragma unroll 4
        for (int k = c & ~3; k < B; k += 4) {
            const float4 f = *reinterpret_cast<const float4*>(low + k);
#pragma unroll
            for (int e = 0; e < 4; ++e) add(acc, (&f.x)[e], L + (k + e) * DC_LD + c);
        }
#pragma unroll
        for (int i = 0; i < COLS / 2; i += 2)
            *reinterpret_cast<float4*>(temp + r * DC_LD + 2 * i) = make_float4(acc[i].x, acc[i].y, acc[i + 1].x, acc[i + 1].y);
    }
    __syncthreads();
    if (live) {
#pragma unroll
        for (int i = 0; i < COLS / 2; ++i) acc[i] = make_float2(0.f, 0.f);
#pragma unroll 4
        for (int k = 0; k < B; k += 4) {
            const float4 f = *reinterpret_cast<const float4*>(low + B + k);
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (k + e <= r) add(acc, -(&f.x)[e], temp + (k + e) * DC_LD);
        }
    }
    __syncthreads();
    if (live) {
#pragma unroll
        for (int i = 0; i < COLS / 2; i += 2) {
            *reinterpret_cast<float4*>(low + c + 2 * i) = make_float4(acc[i].x, acc[i].y, acc[i + 1].x, acc[i + 1].y);
            *reinterpret_cast<float4*>(temp + r * DC_LD + 2 * i) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
    __syncthreads();
}

// T and G of one chunk and the heads of one q/k head, two heads at a time, four warps each; gridDim.z blocks share the pairs of heads.
template <int D>
__global__ void __launch_bounds__(256, 3)
delta_chunk_prepare_kernel(const DeltaChunks m) {
    extern __shared__ __align__(128) uint8_t prep_smem[];
    constexpr int TILE = DC_T * D * 2, MAT = DC_T * DC_LD * 4;
    float* kk = reinterpret_cast<float*>(prep_smem);
    float* qk = kk + DC_T * DC_LD;
    uint8_t* rest = prep_smem + 2 * MAT;       // the tiles of k and q, then a matrix of each head
    __shared__ double half_s[2];
    // a token's logarithm, summed, as two floats (their differences are as exact as 64-bit ones); beta |k|^-1; scale |q|^-1
    __shared__ float4 row_s[2][DC_T];
    __shared__ float2 cum_s[2][DC_T];
    __shared__ float rk_s[DC_T], rq_s[DC_T], beta_s[2][DC_T];
    pdl_launch_dependents();
    pdl_wait();
    const int slot = blockIdx.x, kh = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const Chunk64 at = chunk_of(m.cu_seqlens, m.n_seqs, slot);
    const int first = at.first, nt = at.nt;
    if (nt <= 0) return;
    const __nv_bfloat16* rows = m.qkv + (size_t)first * m.stride;
    const uint32_t kt = shared_u32(rest), qt = kt + TILE;
#pragma unroll
    for (int i = tid; i < DC_T * (D / 8); i += 256) {
        const int t = i / (D / 8), c = i % (D / 8);
        const __nv_bfloat16* src = rows + (t < nt ? (int64_t)t * m.stride : 0) + kh * D + c * 8;
        cp_async16(kt + tile_off<D>(t, c), src + m.k_off, t < nt);
        cp_async16(qt + tile_off<D>(t, c), src + m.q_off, t < nt);
    }
    cp_async_commit();
    // meanwhile the decays' logarithms and beta of the first two heads
    const int per = m.H / m.K, which = warp >> 2, quarter = warp & 3, t = tid & 63;
    double la = 0.0;
    float beta = 0.f;
    auto gates = [&](int r) {
        la = 0.0;
        beta = 0.f;
        if (r >= per || t >= nt || quarter >= 2) return;
        const int h = kh * per + r;
        const float z = m.za[(size_t)(first + t) * m.za_stride + h] + m.bias[h];
        // (a decay of 0 keeps a finite logarithm: differences of two infinite ones would be NaN)
        la = -(double)m.A[h] * (double)(z > 20.f ? z : log1pf(expf(z)));
        la = la < -1e6 ? -1e6 : la;
        beta = 1.0f / (1.0f + expf(-m.zb[(size_t)(first + t) * m.zb_stride + h]));
    };
    const int r_first = 2 * blockIdx.z;
    gates(r_first + which);
    cp_async_wait<0>();
    __syncthreads();
    {   // lengths: four threads a token
        const int i = tid >> 2;
        float sk = 0.f, sq = 0.f;
#pragma unroll
        for (int c = 0; c < D / 32; ++c) {
            const uint32_t off = tile_off<D>(i, c * 4 + (tid & 3));
            const uint4 kv = *reinterpret_cast<const uint4*>(rest + off), qv = *reinterpret_cast<const uint4*>(rest + TILE + off);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const uint32_t a = (&kv.x)[e], b = (&qv.x)[e];
                const float k0 = __uint_as_float(a << 16), k1 = __uint_as_float(a & 0xffff0000u);
                const float q0 = __uint_as_float(b << 16), q1 = __uint_as_float(b & 0xffff0000u);
                sk = fmaf(k1, k1, fmaf(k0, k0, sk));
                sq = fmaf(q1, q1, fmaf(q0, q0, sq));
            }
        }
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) {
            sk += __shfl_xor_sync(0xffffffffu, sk, o);
            sq += __shfl_xor_sync(0xffffffffu, sq, o);
        }
        if ((tid & 3) == 0) {
            rk_s[i] = 1.0f / sqrtf(sk + 1e-6f);
            rq_s[i] = 1.0f / sqrtf(sq + 1e-6f) * m.q_scale;
        }
    }
    for (int n = warp; n < 20; n += 8) lower_block<D>(n < 10 ? kk : qk, n < 10 ? kt : qt, kt, n % 10, lane);
    float* L = reinterpret_cast<float*>(rest) + which * DC_T * DC_LD;
    for (int r0 = r_first; r0 < per; r0 += 2 * gridDim.z) {
        const int h = kh * per + r0 + which;
        const bool live = r0 + which < per;
        if (r0 > r_first) gates(r0 + which);
        if (quarter < 2) {
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const double up = __shfl_up_sync(0xffffffffu, la, o);
                if (lane >= o) la += up;
            }
            if (t == 31) half_s[which] = la;
        }
        __syncthreads();                       // (also: the products above are written, the round before is done with L)
        if (quarter < 2) {
            if (t >= 32) la += half_s[which];
            const float2 cum = make_float2((float)la, (float)(la - (double)(float)la));
            cum_s[which][t] = cum;
            row_s[which][t] = make_float4(cum.x, cum.y, beta * rk_s[t], rq_s[t]);
            if (t == DC_T - 1) half_s[which] = la;
            beta_s[which][t] = beta;
        }
        __syncthreads();
        uint8_t* mats = m.mats + ((size_t)slot * m.H + h) * DC_MATS;
        if (live) {
            if (quarter < 2) {
                const double end = half_s[which];
                float* f = m.factors + ((size_t)slot * m.H + h) * DC_FACTORS * DC_T;
                const float gone = expf((float)la);
                f[DC_K * DC_T + t] = gone * rk_s[t];
                f[DC_Q * DC_T + t] = gone * rq_s[t];
                f[DC_W * DC_T + t] = expf((float)(end - la)) * rk_s[t];
                if (t == 0) f[DC_END * DC_T] = expf((float)end);
            }
#pragma unroll
            for (int n = 0; n < DC_STEPS; ++n) {
                const int2 at = triangle_step(n, quarter, lane);
                const int c = at.y & (DC_T - 2);
                const float4 ri = row_s[which][at.x];
                const float2 a0 = cum_s[which][c], a1 = cum_s[which][c + 1];
                const float2 rk = *reinterpret_cast<const float2*>(rk_s + c);
                const float2 ki = *reinterpret_cast<const float2*>(kk + at.x * DC_LD + c);
                const float2 qi = *reinterpret_cast<const float2*>(qk + at.x * DC_LD + c);
                const float e0 = expf((ri.x - a0.x) + (ri.y - a0.y)) * rk.x, e1 = expf((ri.x - a1.x) + (ri.y - a1.y)) * rk.y;
                const float2 l = make_float2(c < at.x ? e0 * ri.z * ki.x : 0.f, c + 1 < at.x ? e1 * ri.z * ki.y : 0.f);
                if (at.y >= DC_T) continue;
                *reinterpret_cast<float2*>(L + at.x * DC_LD + c) = l;
                store_parts(mats + 3 * DC_PART, at, c <= at.x ? e0 * ri.w * qi.x : 0.f, c < at.x ? e1 * ri.w * qi.y : 0.f);
            }
        }
        __syncthreads();
        // L becomes (1 + L)^-1: the blocks of 16 on the diagonal column by column, then twice the block left of two that are done,
        // -T22 (L21 T11), the inner product by way of the block above the diagonal
        if (live && quarter < 2) {
            float* at = L + (t & ~15) * (DC_LD + 1);
            const int c = t & 15;
            float2 x[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) x[i] = make_float2(0.f, 0.f);
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                float2 p = make_float2(0.f, 0.f), q = p;
#pragma unroll
                for (int k = 0; k < i; k += 4) {
                    const float4 l = *reinterpret_cast<const float4*>(at + i * DC_LD + k);
                    p = fma2(make_float2(l.x, l.y), x[k / 2], p);
                    q = fma2(make_float2(l.z, l.w), x[k / 2 + 1], q);
                }
                const float v = i == c ? 1.f : -((p.x + p.y) + (q.x + q.y));
                if (i & 1) x[i / 2].y = v;
                else x[i / 2].x = v;
            }
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 16; ++i) at[i * DC_LD + c] = i & 1 ? x[i / 2].y : x[i / 2].x;
        }
        __syncthreads();
        join_blocks<16, 4>(L + (quarter >> 1) * 32 * (DC_LD + 1), lane & 15, (quarter & 1) * 8 + (lane >> 4) * 4, live);
        join_blocks<32, 8>(L, lane, quarter * 8, live);
        if (live) {
#pragma unroll
            for (int n = 0; n < DC_STEPS; ++n) {
                const int2 at = triangle_step(n, quarter, lane);
                if (at.y >= DC_T) continue;
                const float2 v = *reinterpret_cast<const float2*>(L + at.x * DC_LD + at.y);
                const float2 b = *reinterpret_cast<const float2*>(&beta_s[which][at.y]);
                // (above the diagonal: 0 whatever beta is)
                store_parts(mats, at, at.y <= at.x ? v.x * b.x : 0.f, at.y < at.x ? v.y * b.y : 0.f);
            }
        }
    }
}

__device__ __forceinline__ bool dc_odd(float x) { return !(fabsf(x) <= 3.402823466e38f); }

// (high, rest, rest) of two neighbouring tiles += left (three parts of 16 rows x 16 tokens) times the 16 x 16 block (rows, columns) of a
// matrix of three parts, turned round. The three chains of each tile leave a product's latency between two of one chain.
struct DcSums {
    float hi[2][4], lo[2][4], mid[2][4];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int q = 0; q < 2; ++q)
#pragma unroll
            for (int e = 0; e < 4; ++e) hi[q][e] = lo[q][e] = mid[q][e] = 0.f;
    }
    __device__ __forceinline__ float sum(int q, int e) const { return hi[q][e] + (mid[q][e] + lo[q][e]); }
};
__device__ __forceinline__ void dc_six(DcSums& c, const uint32_t (&a)[3][4], uint32_t mat, int block_row, int block_col, int lane) {
    const uint32_t at = mat + tile_off<DC_T>(block_row * 16 + (lane & 7) + (lane >> 4) * 8, block_col * 2 + ((lane >> 3) & 1));
    uint32_t b[3][4];
#pragma unroll
    for (int p = 0; p < 3; ++p) ldmatrix_x4(b[p], at + p * DC_PART);
    mma16816(c.hi[0], a[0], b[0][0], b[0][1]);
    mma16816(c.hi[1], a[0], b[0][2], b[0][3]);
    mma16816(c.lo[0], a[2], b[0][0], b[0][1]);
    mma16816(c.lo[1], a[2], b[0][2], b[0][3]);
    mma16816(c.mid[0], a[1], b[0][0], b[0][1]);
    mma16816(c.mid[1], a[1], b[0][2], b[0][3]);
    mma16816(c.lo[0], a[1], b[1][0], b[1][1]);
    mma16816(c.lo[1], a[1], b[1][2], b[1][3]);
    mma16816(c.mid[0], a[0], b[1][0], b[1][1]);
    mma16816(c.mid[1], a[0], b[1][2], b[1][3]);
    mma16816(c.lo[0], a[0], b[2][0], b[2][1]);
    mma16816(c.lo[1], a[0], b[2][2], b[2][3]);
}

// Shared memory of the walk (bytes): tiles, then what warps hand to each other in the registers' own layout ([..][lane] 16 bytes):
// S's parts, a state warp's half of P, the parts of U and of U diag(A_end / A); the first token of a row that is not finite.
template <int D, int PAIRS>
struct DcSmem {
    static constexpr int TILE = DC_T * D * 2, VROW = PAIRS * 32 + 16;
    static constexpr int K = 0, Q = K + 2 * TILE, T = Q + TILE, G = T + 3 * DC_PART, F = G + 3 * DC_PART;
    static constexpr int S = F + 2 * DC_FACTORS * DC_T * 4, P = S + PAIRS * (D / 16) * 3 * 512, U = P + PAIRS * 2 * 8 * 512;
    static constexpr int W = U + PAIRS * 4 * 3 * 512, ODD = W + PAIRS * 4 * 3 * 512, V = ODD + PAIRS * 2 * 16 * 4;
    static constexpr int ALL = V + DC_T * VROW;
};

// Four warps per 16 rows of V: two carry the state (each half of D's columns, and half of the chunk's tokens of U), two write the
// outputs (half of the tokens each) one barrier behind them, and fetch the tiles.
template <int D, int PAIRS>
__global__ void __launch_bounds__(128 * PAIRS, 1)
delta_chunk_walk_kernel(const DeltaChunks m) {
    using Z = DcSmem<D, PAIRS>;
    constexpr int LOADERS = 64 * PAIRS, DH = D / 2, KS = DH / 16, NS = DH / 8, COLS = 16 * PAIRS;
    extern __shared__ __align__(128) uint8_t walk_smem[];
    const uint32_t base = shared_u32(walk_smem);
    pdl_launch_dependents();
    pdl_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, pair = (warp % (2 * PAIRS)) >> 1, half = warp & 1;
    const int c0 = blockIdx.x * COLS, h = blockIdx.y, s = blockIdx.z, kh = h / (m.H / m.K);
    const int begin = m.cu_seqlens[s], len = m.cu_seqlens[s + 1] - begin;
    if (len <= 0) return;
    const int n_chunks = (len + DC_T - 1) / DC_T;
    const int row = lane >> 2, tok = 2 * (lane & 3);            // the accumulators' row (and row + 8) and first token of eight
    const int v0 = c0 + pair * 16 + row;
    const uint32_t b_row = (lane & 7) + (lane >> 4) * 8, b_chunk = (lane >> 3) & 1;      // ldmatrix rows of a right operand
    uint8_t* const s_parts = walk_smem + Z::S + pair * (D / 16) * 3 * 512 + lane * 16;
    uint8_t* const u_parts = walk_smem + Z::U + pair * 4 * 3 * 512 + lane * 16;
    uint8_t* const w_parts = walk_smem + Z::W + pair * 4 * 3 * 512 + lane * 16;
    int* const odd_at = reinterpret_cast<int*>(walk_smem + Z::ODD) + pair * 32;          // [half][16 rows]
    const float nan = __int_as_float(0x7fffffff);

    if (warp >= 2 * PAIRS) {
        const int tid = threadIdx.x - 64 * PAIRS, slot0 = begin / DC_T + s;
        const __nv_bfloat16* rows = m.qkv + (size_t)begin * m.stride;
        auto load_rows = [&](uint32_t tile, int col, int j) {
            const __nv_bfloat16* src = rows + (size_t)j * DC_T * m.stride + col;
            const int nt = len - j * DC_T;
#pragma unroll
            for (int i = tid; i < DC_T * (D / 8); i += LOADERS) {
                const int t = i / (D / 8), c = i % (D / 8);
                cp_async16(tile + tile_off<D>(t, c), src + (t < nt ? (int64_t)t * m.stride : 0) + c * 8, t < nt);
            }
        };
        auto load_mat = [&](uint32_t dst, int j, int part) {
            const uint8_t* src = m.mats + ((size_t)(slot0 + j) * m.H + h) * DC_MATS + part * DC_PART;
#pragma unroll
            for (int i = tid; i < 3 * DC_PART / 16; i += LOADERS) cp_async16(dst + i * 16, src + i * 16, true);
        };
        auto load_k = [&](int j) { load_rows(base + Z::K + (j & 1) * Z::TILE, m.k_off + kh * D, j); };
        auto load_rest = [&](int j) {                           // all that a chunk needs from its first barrier on
            load_rows(base + Z::Q, m.q_off + kh * D, j);
            load_mat(base + Z::T, j, 0);
            const float* f = m.factors + ((size_t)(slot0 + j) * m.H + h) * DC_FACTORS * DC_T;
            const uint32_t dst = base + Z::F + (j & 1) * DC_FACTORS * DC_T * 4;
            for (int i = tid; i < DC_FACTORS * DC_T / 4; i += LOADERS) cp_async16(dst + i * 16, f + i * 4, true);
            const __nv_bfloat16* v = rows + (size_t)j * DC_T * m.stride + m.v_off + h * m.V + c0;
            const int nt = len - j * DC_T;
#pragma unroll
            for (int i = tid; i < DC_T * (COLS / 8); i += LOADERS) {
                const int t = i / (COLS / 8), c = i % (COLS / 8);
                cp_async16(base + Z::V + t * Z::VROW + c * 16, v + (t < nt ? (int64_t)t * m.stride : 0) + c * 8, t < nt);
            }
        };
        load_k(0);
        load_rest(0);
        cp_async_commit();
        cp_async_wait<0>();
        dc_sync();
        const int HV = m.H * m.V;
        float* y = m.y + (size_t)begin * HV + h * m.V + v0;
        // the tokens of this warp: blocks of 16 tokens 0 and 3, or 1 and 2 (the same number of blocks left of the diagonal)
        for (int j = 0; j < n_chunks; ++j) {
            const float* f = reinterpret_cast<const float*>(walk_smem + Z::F + (j & 1) * DC_FACTORS * DC_T * 4);
            float hi[4][4], hi2[4][4], lo[4][4];                // (high parts in two chains: half the sums that are cut off)
            dc_zero(hi);
            dc_zero(hi2);
            dc_zero(lo);
            dc_sync();                                          // S's parts, q, T, the values and the factors are there
            if (j + 1 < n_chunks) load_k(j + 1);
            load_mat(base + Z::G, j, 3);
            cp_async_commit();
#pragma unroll
            for (int ks = 0; ks < D / 16; ++ks) {
                uint32_t a[3][4], b[4], b2[4];
                dc_take(a, s_parts + ks * 3 * 512);
                ldmatrix_x4(b, base + Z::Q + tile_off<D>(half * 16 + b_row, ks * 2 + b_chunk));
                ldmatrix_x4(b2, base + Z::Q + tile_off<D>((3 - half) * 16 + b_row, ks * 2 + b_chunk));
                float(&top)[4][4] = ks & 1 ? hi2 : hi;
                dc_three(top[0], top[1], lo[0], lo[1], a, b);
                dc_three(top[2], top[3], lo[2], lo[3], a, b2);
            }
            float out[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int t = (i < 2 ? half : 3 - half) * 16 + (i & 1) * 8 + tok;
                const float2 w = *reinterpret_cast<const float2*>(f + DC_Q * DC_T + t);
#pragma unroll
                for (int e = 0; e < 4; ++e) out[i][e] = (e & 1 ? w.y : w.x) * (hi[i][e] + hi2[i][e] + lo[i][e]);
            }
            cp_async_wait<0>();
            dc_sync();                                          // U's parts, G and the next k are there
            if (j + 1 < n_chunks) load_rest(j + 1);
            cp_async_commit();
            DcSums c[2];
            c[0].clear();
            c[1].clear();
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (k > 3 - half) continue;
                uint32_t a[3][4];
                dc_take(a, u_parts + k * 3 * 512);
                dc_six(c[1], a, base + Z::G, 3 - half, k, lane);
                if (k <= half) dc_six(c[0], a, base + Z::G, half, k, lane);
            }
            const int odd0 = min(odd_at[row], odd_at[16 + row]), odd1 = min(odd_at[row + 8], odd_at[24 + row]);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int t = (i < 2 ? half : 3 - half) * 16 + (i & 1) * 8 + tok;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    out[i][e] += c[i >> 1].sum(i & 1, e);
                    if (t + (e & 1) >= (e < 2 ? odd0 : odd1)) out[i][e] = nan;
                }
                float* dst = y + (size_t)(j * DC_T + t) * HV;
                if (j * DC_T + t < len) dst[0] = out[i][0], dst[8] = out[i][2];
                if (j * DC_T + t + 1 < len) dst[HV] = out[i][1], dst[HV + 8] = out[i][3];
            }
            cp_async_wait<0>();
        }
        return;
    }

    float* st = m.state + ((size_t)TK_SLOT(TK_K_DELTA_CHUNKS, m.seq_slot[s]) * m.H + h) * m.V * D + half * DH + tok;
    float S[NS][4];
    const bool carried = m.seq_ctx[s] > 0;
#pragma unroll
    for (int n = 0; n < NS; ++n) {
        float2 a = make_float2(0.f, 0.f), b = a;
        if (carried) {
            a = *reinterpret_cast<const float2*>(st + (size_t)v0 * D + n * 8);
            b = *reinterpret_cast<const float2*>(st + (size_t)(v0 + 8) * D + n * 8);
        }
        S[n][0] = a.x, S[n][1] = a.y, S[n][2] = b.x, S[n][3] = b.y;
    }
    float4* mine = reinterpret_cast<float4*>(walk_smem + Z::P + warp * 8 * 512) + lane;
    const float4* theirs = reinterpret_cast<const float4*>(walk_smem + Z::P + (warp ^ 1) * 8 * 512) + lane;
    dc_sync();

    for (int j = 0; j < n_chunks; ++j) {
        const uint32_t kt = base + Z::K + (j & 1) * Z::TILE;
        const float* f = reinterpret_cast<const float*>(walk_smem + Z::F + (j & 1) * DC_FACTORS * DC_T * 4);
        // this warp's half of the sums of P
        float P[8][4];
        {
            float lo[8][4];
            dc_zero(P);
            dc_zero(lo);
#pragma unroll
            for (int ks = 0; ks < KS; ++ks) {
                uint32_t a[3][4], b[4][4];
                dc_cut(a, S[2 * ks], S[2 * ks + 1]);
                dc_give(s_parts + (half * KS + ks) * 3 * 512, a);
#pragma unroll
                for (int np = 0; np < 4; ++np)
                    ldmatrix_x4(b[np], kt + tile_off<D>(np * 16 + b_row, half * (DH / 8) + ks * 2 + b_chunk));
#pragma unroll
                for (int np = 0; np < 4; ++np) dc_three(P[2 * np], P[2 * np + 1], lo[2 * np], lo[2 * np + 1], a, b[np]);
            }
#pragma unroll
            for (int n = 0; n < 8; ++n) {
#pragma unroll
                for (int e = 0; e < 4; ++e) P[n][e] += lo[n][e];
                mine[n * 32] = make_float4(P[n][0], P[n][1], P[n][2], P[n][3]);
            }
        }
        dc_sync();
        // R, then this warp's tokens of U: blocks of 16 tokens 0 and 3, or 1 and 2
        int odd0 = DC_T, odd1 = DC_T;                           // the first token of rows row and row + 8 that is not finite
        float probe = 0.f;                                      // stays 0 while every number it has met is finite
#pragma unroll
        for (int np = 0; np < 4; ++np) {
            uint32_t vv[4];                                     // values: (8 tokens, rows 0-7), (rows 8-15), the next 8 tokens
            ldmatrix_x4_trans(vv, base + Z::V + (np * 16 + b_row) * Z::VROW + pair * 32 + b_chunk * 16);
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int n = 2 * np + q;
                const float4 o = theirs[n * 32];
                const float2 w = *reinterpret_cast<const float2*>(f + DC_K * DC_T + n * 8 + tok);
                P[n][0] = fmaf(-w.x, P[n][0] + o.x, __uint_as_float(vv[2 * q] << 16));
                P[n][1] = fmaf(-w.y, P[n][1] + o.y, __uint_as_float(vv[2 * q] & 0xffff0000u));
                P[n][2] = fmaf(-w.x, P[n][2] + o.z, __uint_as_float(vv[2 * q + 1] << 16));
                P[n][3] = fmaf(-w.y, P[n][3] + o.w, __uint_as_float(vv[2 * q + 1] & 0xffff0000u));
#pragma unroll
                for (int e = 0; e < 4; ++e) probe = fmaf(P[n][e], 0.f, probe);
            }
        }
        if (__any_sync(0xffffffffu, probe != 0.f)) {
#pragma unroll
            for (int n = 0; n < 8; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (dc_odd(P[n][e])) {
                        P[n][e] = 0.f;
                        int& first = e < 2 ? odd0 : odd1;
                        first = min(first, n * 8 + tok + (e & 1));
                    }
        }
        uint32_t own[2][3][4];                                  // the parts of this warp's two blocks of U diag(A_end / A)
        {
            DcSums c[2];
            c[0].clear();
            c[1].clear();
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (k > 3 - half) continue;
                uint32_t a[3][4];
                dc_cut(a, P[2 * k], P[2 * k + 1]);
                dc_six(c[1], a, base + Z::T, 3 - half, k, lane);
                if (k <= half) dc_six(c[0], a, base + Z::T, half, k, lane);
            }
            float hi[4][4];
            probe = 0.f;
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    hi[i][e] = c[i >> 1].sum(i & 1, e);
                    probe = fmaf(hi[i][e], 0.f, probe);
                }
            if (__any_sync(0xffffffffu, probe != 0.f || odd0 < DC_T || odd1 < DC_T)) {
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (dc_odd(hi[i][e])) {
                            hi[i][e] = 0.f;
                            int& first = e < 2 ? odd0 : odd1;
                            first = min(first, (i < 2 ? half : 3 - half) * 16 + (i & 1) * 8 + tok + (e & 1));
                        }
#pragma unroll
                for (int o = 1; o < 4; o <<= 1) {
                    odd0 = min(odd0, __shfl_xor_sync(0xffffffffu, odd0, o));
                    odd1 = min(odd1, __shfl_xor_sync(0xffffffffu, odd1, o));
                }
            }
            if ((lane & 3) == 0) {
                odd_at[half * 16 + row] = odd0;
                odd_at[half * 16 + row + 8] = odd1;
            }
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int k = i ? 3 - half : half;
                uint32_t a[3][4];
                dc_cut(a, hi[2 * i], hi[2 * i + 1]);
                dc_give(u_parts + k * 3 * 512, a);
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const float2 w = *reinterpret_cast<const float2*>(f + DC_W * DC_T + k * 16 + q * 8 + tok);
                    float(&u)[4] = hi[2 * i + q];
                    u[0] *= w.x, u[1] *= w.y, u[2] *= w.x, u[3] *= w.y;
                }
                dc_cut(own[i], hi[2 * i], hi[2 * i + 1]);
                dc_give(w_parts + k * 3 * 512, own[i]);
            }
        }
        const float end = f[DC_END * DC_T];
        dc_sync();
        // what the chunk adds to this warp's columns of S
        float hi[NS][4], hi2[NS][4], lo[NS][4];
        dc_zero(hi);
        dc_zero(hi2);
        dc_zero(lo);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int k = i == 0 ? half : i == 1 ? 3 - half : i == 2 ? 1 - half : 2 + half;
            uint32_t b[NS / 2][4];
            if (i >= 2) dc_take(own[i - 2], w_parts + k * 3 * 512);
#pragma unroll
            for (int np = 0; np < NS / 2; ++np)
                ldmatrix_x4_trans(b[np], kt + tile_off<D>(k * 16 + (lane & 15), half * (DH / 8) + np * 2 + (lane >> 4)));
#pragma unroll
            for (int np = 0; np < NS / 2; ++np) dc_three((i & 1 ? hi2 : hi)[2 * np], (i & 1 ? hi2 : hi)[2 * np + 1], lo[2 * np], lo[2 * np + 1], own[i & 1], b[np]);
        }
        odd0 = min(odd0, odd_at[(half ^ 1) * 16 + row]);
        odd1 = min(odd1, odd_at[(half ^ 1) * 16 + row + 8]);
#pragma unroll
        for (int n = 0; n < NS; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) S[n][e] = (e < 2 ? odd0 : odd1) < DC_T ? nan : fmaf(end, S[n][e], hi[n][e] + hi2[n][e] + lo[n][e]);
    }
#pragma unroll
    for (int n = 0; n < NS; ++n) {
        *reinterpret_cast<float2*>(st + (size_t)v0 * D + n * 8) = make_float2(S[n][0], S[n][1]);
        *reinterpret_cast<float2*>(st + (size_t)(v0 + 8) * D + n * 8) = make_float2(S[n][2], S[n][3]);
    }
}

template <int D, int PAIRS>
cudaError_t dc_walk(const DeltaChunks& m, cudaStream_t stream) {
    constexpr int smem = DcSmem<D, PAIRS>::ALL;
    auto kernel = delta_chunk_walk_kernel<D, PAIRS>;
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    return tk_launch_after(kernel, dim3(m.V / (16 * PAIRS), m.H, m.n_seqs), dim3(128 * PAIRS), smem, stream, m);
}

template <int D>
void dc_launch(const DeltaChunks& m, int slots, int sm_count, cudaStream_t stream) {
    constexpr int TILE = DC_T * D * 2, MAT = DC_T * DC_LD * 4, smem = 2 * MAT + (2 * TILE > 2 * MAT ? 2 * TILE : 2 * MAT);
    auto prepare = delta_chunk_prepare_kernel<D>;
    cudaFuncSetAttribute(prepare, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    // while three blocks an SM are not reached, the pairs of heads of a q/k head have blocks of their own, each with the products of k
    // and q over again (32 heads over 4: 64 tokens 31.9 us by one block, 18.5 by four; token by token 22.6)
    const int pairs = (m.H / m.K + 1) / 2, blocks = slots * m.K;
    const int shared_by = blocks * pairs <= 3 * sm_count ? pairs : blocks < 3 * sm_count ? 3 * sm_count / blocks : 1;
    tk_launch(prepare, dim3(slots, m.K, shared_by), dim3(256), smem, stream, m);
    // 32 rows of V a block, 16 while those blocks all find an SM of their own (one sequence of 512 tokens, 16 heads of 64 x 64)
    if ((int64_t)m.V / 16 * m.H * m.n_seqs <= sm_count) dc_walk<D, 1>(m, stream);
    else dc_walk<D, 2>(m, stream);
}
}  // namespace

// Words of scratch of a step chunk by chunk, or 0: not taken. A chunk a sequence pays for the first kernel with heads of 128 (16 heads
// over 8: one sequence of 64 tokens 15.1 us, 17.7 token by token; four 23.5 and 28.4; 16 of 100 80 and 126) and with one
// sequence of heads of 64 (64 tokens 13.3 and 15.1); several sequences of heads of 64 are walked side by side until they have
// two (four of 64 20.1 against 16.4, of 100 22.6 and 22.5, of 300 30.8 and 52.4).
TK_API int tk_delta_chunks_scratch(int tokens, int n_seqs, int H, int K, int D, int V) {
    if ((D != 64 && D != 128) || V % 32 != 0 || n_seqs <= 0 || n_seqs > 65535 || H > 65535) return 0;
    if (tokens < (int64_t)DC_T * n_seqs * (D == 64 && n_seqs > 1 ? 2 : 1)) return 0;
    const int64_t words = ((int64_t)tokens / DC_T + n_seqs) * H * DC_WORDS;
    return words * 4 <= (int64_t)512 << 20 ? (int)words : 0;
}

// The delta rule with a decay per head over bfloat16 rows with unit q and k (tk_linmem_scan's arguments); rows, offsets and bases whole
// 16-byte pieces. scratch: what tk_delta_chunks_scratch says, 16-byte aligned.
TK_API int tk_delta_chunks(const void* qkv, int64_t stride, int q_off, int k_off, int v_off, const float* zb, int64_t zb_stride,
                           const float* za, int64_t za_stride, const float* bias, const float* A, float* state,
                           const int* cu_seqlens, const int* seq_ctx, const int* seq_slot, int n_seqs, int tokens, float* y,
                           float* scratch, int H, int K, int D, int V, float q_scale, int sm_count, cudaStream_t stream) {
    TK_CHECK_ARG(H > 0 && K > 0 && H % K == 0, "delta chunks: %d heads over %d q/k heads", H, K);
    TK_CHECK_ARG(tk_delta_chunks_scratch(tokens, n_seqs, H, K, D, V) > 0 && scratch != nullptr,
                 "delta chunks: %d tokens in %d sequences, heads of %d x %d", tokens, n_seqs, D, V);
    TK_CHECK_ARG(stride % 8 == 0 && q_off % 8 == 0 && k_off % 8 == 0 && v_off % 8 == 0 &&
                     (((uintptr_t)qkv | (uintptr_t)scratch | (uintptr_t)state) & 15) == 0,
                 "delta chunks: rows must be whole 16-byte pieces");
    const int slots = tokens / DC_T + n_seqs;
    const DeltaChunks m{(const __nv_bfloat16*)qkv, stride, q_off, k_off, v_off, zb, zb_stride, za, za_stride, bias, A, state,
                        cu_seqlens, seq_ctx, seq_slot, n_seqs, y, H, K, V, q_scale, reinterpret_cast<uint8_t*>(scratch),
                        scratch + (size_t)slots * H * (DC_MATS / 4)};
    if (D == 64) dc_launch<64>(m, slots, sm_count, stream);
    else dc_launch<128>(m, slots, sm_count, stream);
    TK_CHECK_LAUNCH("delta_chunks");
    return 0;
}
