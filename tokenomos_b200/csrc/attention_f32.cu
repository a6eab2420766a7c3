// Paged attention of the true 32-bit path for heads of 64: 32-bit multiply-adds, scores, softmax and sums on the CUDA
// cores (every mask of attention_generic.cu but a sink and kept first positions, no cap and no bias; anything else goes
// there).
//
// Prompt portions: a block of 256 threads owns 64 rows ((token, query head of the group) pairs that share a KV head) and
// walks their keys 64 at a time. Bound by the multiply-adds, so the split is the one that feeds them: a thread holds 4 x 4
// scores, then 4 x 4 outputs, as pairs (two halves of the inner dimension, packed multiply-adds), and both products read
// their operands as rows along the inner dimension, 16 bytes for four steps of it: 8 shared loads for 64 multiply-adds. For
// that the values are stored turned round ([column][key]). Rows of 68 floats keep the 16-byte reads free of conflicts. Two
// blocks share an SM, so that one's loads and softmax run under the other's products.
//
// Single tokens: bound by the stream of keys and values. A half-warp takes whole keys (16 lanes x 16 bytes), four in
// flight with their values, for all heads of the group; the keys of a token are shared out over `nsplit` blocks and their
// eight half-warps, each with a softmax of its own, merged in a fixed order in the block, then by a second kernel.
//
// An attention layer of 16 / 8 heads on a prompt of 1,000 tokens: 193 us with the prompt kernel, 734 us with the general one
// (16 rows a block, one multiply-add a shared load); of 32 / 8 heads decoding behind about 300 to 3,000 positions, at one
// to 64 requests, the general kernel walked a token's keys in one block of 16 rows.
#include <math.h>

#include "packed.cuh"

namespace {

constexpr int F_D = 64, F_ROWS = 64, F_KEYS = 64, F_LD = F_D + 4, F_THREADS = 256;

__global__ void __launch_bounds__(F_THREADS, 2)
attn32_prefill_kernel(const float* q, const float* kv_pool, float* out, const int* positions, const int* tok_seq,
                      const int* block_table, int bt_stride, const int* tile_tok0, const int* tile_ntok, int H, int Hkv,
                      int P, int window, float scale) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float smem[];
    float* Qs = smem;                        // [row][d]
    float* Ks = Qs + F_ROWS * F_LD;          // [key][d]
    float* Vt = Ks + F_KEYS * F_LD;          // [d][key]
    float* Ps = Vt + F_D * F_LD;             // [row][key]
    __shared__ int64_t key_at[F_KEYS];       // where a key's row begins in the pool (-1: no such key)
    const int G = H / Hkv, kvh = blockIdx.x % Hkv;
    // the longest tiles of a list come last in it: they are begun first
    const int tile = gridDim.x / Hkv - 1 - blockIdx.x / Hkv;
    const int tok0 = tile_tok0[tile], ntok = tile_ntok[tile];
    if (ntok <= 0) return;                   // an unused entry of a fixed-length tile list (captured steps)
    const int rows = ntok * G, seq = tok_seq[tok0], tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;
    for (int i = tid; i < F_ROWS * (F_D / 4); i += F_THREADS) {
        const int r = i / (F_D / 4), c = i % (F_D / 4) * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < rows) v = *reinterpret_cast<const float4*>(q + ((size_t)(tok0 + r / G) * H + kvh * G + r % G) * F_D + c);
        *reinterpret_cast<float4*>(Qs + r * F_LD + c) = v;
    }
    int pos[4], seen[4];                     // this thread's rows: their position and the first one they see
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = ty * 4 + i;
        pos[i] = r < rows ? positions[tok0 + r / G] : -1;
        seen[i] = first_seen(pos[i], window);
    }
    const int lo = first_seen(positions[tok0], window), last = positions[tok0 + ntok - 1];
    float m[4], l[4];
    float2 o[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        m[i] = -INFINITY;
        l[i] = 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) o[i][j] = make_float2(0.f, 0.f);
    }
    const int64_t v_off = (int64_t)Hkv * P * F_D;
    for (int j0 = lo; j0 <= last; j0 += F_KEYS) {
        __syncthreads();                     // the tile before is done with
        if (tid < F_KEYS) {
            const int j = j0 + tid;
            int64_t at = -1;
            if (j <= last) {
                const int page = TK_PAGE(TK_K_ATTN_GENERIC, block_table[(size_t)seq * bt_stride + j / P]);
                at = (((int64_t)page * 2 * Hkv + kvh) * P + j % P) * F_D;
            }
            key_at[tid] = at;
        }
        __syncthreads();
        float4 kv[4], vv[4];
        float bad = 0.f;                     // NaN once a value is not finite
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            // keys: 16 lanes a row; values: a lane a row, so that its four columns turn round without conflicts
            const int i = tid + e * F_THREADS;
            const int64_t ka = key_at[i >> 4], va = key_at[i & 63];
            kv[e] = vv[e] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (ka >= 0) kv[e] = *reinterpret_cast<const float4*>(kv_pool + ka + (i & 15) * 4);
            if (va >= 0) vv[e] = *reinterpret_cast<const float4*>(kv_pool + va + v_off + (i >> 6) * 4);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int i = tid + e * F_THREADS;
            *reinterpret_cast<float4*>(Ks + (i >> 4) * F_LD + (i & 15) * 4) = kv[e];
            float* turned = Vt + (i >> 6) * 4 * F_LD + (i & 63);
            turned[0] = vv[e].x;
            turned[F_LD] = vv[e].y;
            turned[2 * F_LD] = vv[e].z;
            turned[3 * F_LD] = vv[e].w;
            bad = fmaf(vv[e].x, 0.f, fmaf(vv[e].y, 0.f, fmaf(vv[e].z, 0.f, fmaf(vv[e].w, 0.f, bad))));
        }
        const int guarded = __syncthreads_or(bad != bad);
        float2 s2[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) s2[i][j] = make_float2(0.f, 0.f);
        tile_product<4>(Qs + ty * 4 * F_LD, F_LD, Ks + tx * F_LD, F_LD, F_D, s2);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float s[4], mx = -INFINITY;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int key = j0 + tx + 16 * j;
                s[j] = key <= pos[i] && key >= seen[i] ? (s2[i][j].x + s2[i][j].y) * scale : -INFINITY;
                mx = fmaxf(mx, s[j]);
            }
#pragma unroll
            for (int w = 8; w > 0; w >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, w));
            const float m_new = fmaxf(m[i], mx), m_safe = m_new == -INFINITY ? 0.f : m_new;
            const float alpha = expf(m[i] - m_safe);
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float p = expf(s[j] - m_safe);
                sum += p;
                Ps[(ty * 4 + i) * F_LD + tx + 16 * j] = p;
            }
#pragma unroll
            for (int w = 8; w > 0; w >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, w);
            l[i] = l[i] * alpha + sum;
            m[i] = m_new;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                o[i][j].x *= alpha;
                o[i][j].y *= alpha;
            }
        }
        __syncwarp();                        // a row's weights are written and read by the same half-warp
        if (!guarded) {
            tile_product<4>(Ps + ty * 4 * F_LD, F_LD, Vt + tx * F_LD, F_LD, F_KEYS, o);
            continue;
        }
        // a weight of zero does not hide a value that is not finite: the keys a row sees, and no others
        for (int k = 0; k < F_KEYS; ++k)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (j0 + k > pos[i] || j0 + k < seen[i]) continue;
                const float p = Ps[(ty * 4 + i) * F_LD + k];
#pragma unroll
                for (int j = 0; j < 4; ++j) o[i][j].x = fmaf(p, Vt[(tx + 16 * j) * F_LD + k], o[i][j].x);
            }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = ty * 4 + i;
        if (r >= rows) continue;
        float* dst = out + ((size_t)(tok0 + r / G) * H + kvh * G + r % G) * F_D;
        const float inv = l[i] > 0.f ? 1.0f / l[i] : 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) dst[tx + 16 * j] = (o[i][j].x + o[i][j].y) * inv;
    }
}

template <int G>
__global__ void __launch_bounds__(128)
attn32_decode_kernel(const float* q, const float* kv_pool, float* out, const int* positions, const int* tok_seq,
                     const int* block_table, int bt_stride, const int* tok_index, int H, int Hkv, int P, int window,
                     float scale, int nsplit, float* part_o, float* part_ml) {
    constexpr int U = 4;                     // keys a half-warp has in flight
    pdl_launch_dependents();
    pdl_wait();
    __shared__ __align__(16) float acc_s[8][G][F_D];
    __shared__ float m_s[8][G], l_s[8][G];
    const int n = blockIdx.x, kvh = blockIdx.y, split = blockIdx.z;
    const int tok = tok_index != nullptr ? tok_index[n] : n;
    if (tok < 0) return;                     // an unused entry of a fixed-length list (captured steps)
    const int tid = threadIdx.x, hw = tid >> 4, lane = tid & 15;
    const int pos = positions[tok], lo = first_seen(pos, window);
    const int* table = block_table + (size_t)tok_seq[tok] * bt_stride;
    const int count = pos - lo + 1, per = ((count + nsplit - 1) / nsplit + 8 * U - 1) / (8 * U) * (8 * U);
    const int begin = lo + split * per, end = min(begin + per, pos + 1);
    float4 qv[G];
#pragma unroll
    for (int g = 0; g < G; ++g)
        qv[g] = *reinterpret_cast<const float4*>(q + ((size_t)tok * H + kvh * G + g) * F_D + lane * 4);
    float m[G], l[G];
    float4 acc[G];
#pragma unroll
    for (int g = 0; g < G; ++g) {
        m[g] = -INFINITY;
        l[g] = 0.f;
        acc[g] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    for (int j0 = begin; j0 < end; j0 += 8 * U) {
        float4 k[U], v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int j = j0 + hw + 8 * u;
            k[u] = v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (j < end) {
                const int page = TK_PAGE(TK_K_ATTN_GENERIC, table[j / P]);
                const float* at = kv_pool + (((size_t)page * 2 * Hkv + kvh) * P + j % P) * F_D + lane * 4;
                k[u] = *reinterpret_cast<const float4*>(at);
                v[u] = *reinterpret_cast<const float4*>(at + (size_t)Hkv * P * F_D);
            }
        }
#pragma unroll
        for (int g = 0; g < G; ++g) {
            float s[U], mx = m[g];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                s[u] = fmaf(qv[g].x, k[u].x, fmaf(qv[g].y, k[u].y, fmaf(qv[g].z, k[u].z, qv[g].w * k[u].w)));
#pragma unroll
                for (int w = 8; w > 0; w >>= 1) s[u] += __shfl_xor_sync(0xffffffffu, s[u], w);
                s[u] = j0 + hw + 8 * u < end ? s[u] * scale : -INFINITY;
                mx = fmaxf(mx, s[u]);
            }
            const float safe = mx == -INFINITY ? 0.f : mx, alpha = expf(m[g] - safe);
            m[g] = mx;
            l[g] *= alpha;
            acc[g].x *= alpha, acc[g].y *= alpha, acc[g].z *= alpha, acc[g].w *= alpha;
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const float p = expf(s[u] - safe);
                l[g] += p;
                acc[g].x = fmaf(p, v[u].x, acc[g].x);
                acc[g].y = fmaf(p, v[u].y, acc[g].y);
                acc[g].z = fmaf(p, v[u].z, acc[g].z);
                acc[g].w = fmaf(p, v[u].w, acc[g].w);
            }
        }
    }
#pragma unroll
    for (int g = 0; g < G; ++g) {
        *reinterpret_cast<float4*>(&acc_s[hw][g][lane * 4]) = acc[g];
        if (lane == 0) m_s[hw][g] = m[g], l_s[hw][g] = l[g];
    }
    __syncthreads();
    for (int i = tid; i < G * F_D; i += 128) {
        const int g = i / F_D, c = i % F_D, head = kvh * G + g;
        float M = -INFINITY, L = 0.f, o = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) M = fmaxf(M, m_s[w][g]);
#pragma unroll
        for (int w = 0; w < 8; ++w) {
            const float f = m_s[w][g] == -INFINITY ? 0.f : expf(m_s[w][g] - M);
            L += l_s[w][g] * f;
            o += acc_s[w][g][c] * f;
        }
        if (nsplit == 1) {
            out[((size_t)tok * H + head) * F_D + c] = L > 0.f ? o / L : 0.f;
        } else {
            const size_t base = ((size_t)n * H + head) * nsplit + split;
            part_o[base * F_D + c] = o;
            if (c == 0) part_ml[base * 2] = M, part_ml[base * 2 + 1] = L;
        }
    }
}

__global__ void __launch_bounds__(F_D)
attn32_merge_kernel(const float* part_o, const float* part_ml, float* out, const int* tok_index, int H, int nsplit) {
    pdl_launch_dependents();
    pdl_wait();
    const int n = blockIdx.x, head = blockIdx.y, c = threadIdx.x;
    const int tok = tok_index != nullptr ? tok_index[n] : n;
    if (tok < 0) return;
    const size_t base = ((size_t)n * H + head) * nsplit;
    float M = -INFINITY, L = 0.f, o = 0.f;
    for (int s = 0; s < nsplit; ++s) M = fmaxf(M, part_ml[(base + s) * 2]);
    for (int s = 0; s < nsplit; ++s) {
        const float ms = part_ml[(base + s) * 2], f = ms == -INFINITY ? 0.f : expf(ms - M);
        L += part_ml[(base + s) * 2 + 1] * f;
        o += part_o[(base + s) * F_D + c] * f;
    }
    out[((size_t)tok * H + head) * F_D + c] = L > 0.f ? o / L : 0.f;
}

bool group_taken(int G) { return G == 1 || G == 2 || G == 4 || G == 8; }

}  // namespace

// Whether these kernels take a layer's heads (float32 queries and cache, keys and values of 64).
TK_API int tk_attn_f32_supported(int H, int Hkv, int D) { return D == F_D && Hkv > 0 && H % Hkv == 0 && group_taken(H / Hkv); }

// Tokens of one sequence a prompt tile takes.
TK_API int tk_attn_f32_tokens(int H, int Hkv) { return F_ROWS / (H / Hkv); }

// q, out: float32 [T, H, 64]; kv_pool: float32 [pages, 2, Hkv, P, 64]; tiles of at most tk_attn_f32_tokens tokens of one
// sequence with consecutive positions; window: see first_seen.
TK_API int tk_attn_f32_prefill(const void* q, const void* kv_pool, void* out, const int* positions, const int* tok_seq,
                               const int* block_table, int bt_stride, const int* tile_tok0, const int* tile_ntok, int n_tiles,
                               int H, int Hkv, int P, int window, float scale, cudaStream_t stream) {
    TK_CHECK_ARG(tk_attn_f32_supported(H, Hkv, F_D), "attention (32-bit): %d query heads over %d KV heads", H, Hkv);
    TK_CHECK_ARG(P > 0 && n_tiles >= 0 && (int64_t)n_tiles * Hkv < 0x7fffffff, "attention (32-bit): bad page size or tile count");
    TK_CHECK_ARG((uintptr_t)q % 16 == 0 && (uintptr_t)kv_pool % 16 == 0, "attention (32-bit): 16-byte aligned bases");
    if (n_tiles == 0) return 0;
    const int smem = (2 * F_ROWS + F_KEYS + F_D) * F_LD * (int)sizeof(float);
    cudaFuncSetAttribute(attn32_prefill_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    tk_launch(attn32_prefill_kernel, dim3(n_tiles * Hkv), dim3(F_THREADS), smem, stream, (const float*)q, (const float*)kv_pool,
              (float*)out, positions, tok_seq, block_table, bt_stride, tile_tok0, tile_ntok, H, Hkv, P, window, scale);
    TK_CHECK_LAUNCH("attn_f32_prefill");
    return 0;
}

// Sequences that bring one token: tok_index their rows of q (null: all of them, in order), `nsplit` blocks a (token, KV head);
// scratch: float32 [n, H, nsplit, 66] when nsplit > 1.
TK_API int tk_attn_f32_decode(const void* q, const void* kv_pool, void* out, const int* positions, const int* tok_seq,
                              const int* block_table, int bt_stride, const int* tok_index, int n, int H, int Hkv, int P,
                              int window, float scale, int nsplit, float* scratch, cudaStream_t stream) {
    TK_CHECK_ARG(tk_attn_f32_supported(H, Hkv, F_D), "attention (32-bit): %d query heads over %d KV heads", H, Hkv);
    TK_CHECK_ARG(P > 0 && n >= 0 && nsplit >= 1 && nsplit <= 65535 && (nsplit == 1 || scratch != nullptr),
                 "attention (32-bit): bad page size, count or splits");
    TK_CHECK_ARG((uintptr_t)q % 16 == 0 && (uintptr_t)kv_pool % 16 == 0, "attention (32-bit): 16-byte aligned bases");
    if (n == 0) return 0;
    float *part_o = scratch, *part_ml = scratch + (size_t)n * H * nsplit * F_D;
#define TK_D32(G)                                                                                                        \
    tk_launch(attn32_decode_kernel<G>, dim3(n, Hkv, nsplit), dim3(128), 0, stream, (const float*)q, (const float*)kv_pool, \
              (float*)out, positions, tok_seq, block_table, bt_stride, tok_index, H, Hkv, P, window, scale, nsplit, part_o, \
              part_ml)
    switch (H / Hkv) {
        case 1: TK_D32(1); break;
        case 2: TK_D32(2); break;
        case 4: TK_D32(4); break;
        default: TK_D32(8); break;
    }
#undef TK_D32
    TK_CHECK_LAUNCH("attn_f32_decode");
    if (nsplit > 1) {
        tk_launch(attn32_merge_kernel, dim3(n, H), dim3(F_D), 0, stream, (const float*)part_o, (const float*)part_ml, (float*)out,
                  tok_index, H, nsplit);
        TK_CHECK_LAUNCH("attn_f32_merge");
    }
    return 0;
}
