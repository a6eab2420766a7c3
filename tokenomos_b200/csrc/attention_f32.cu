// Paged attention of the true 32-bit path for heads of 64 (every mask of attention_generic.cu but a sink and kept first
// positions, no cap and no bias; anything else goes there).
//
// Prompt portions: on the tensor cores, 32-bit numbers as three 16-bit parts (parts.cuh; six products of nine, the high
// parts' sums apart from the rest and each tile's joined in 32-bit registers). Four warps own 64 rows ((token, query head of
// the group) pairs that share a KV head), 16 each, and walk their keys 64 at a time: q lies in shared memory in parts as the
// registers take it, keys and values come by cp.async as floats, are taken apart by the thread that fetched them and shared as
// six 16-bit tiles. A tile takes a block 4.5 us, two blocks of an SM 3.4 us each: 384 mma.sync of 8 cycles a warp beside 1,800 other
// instructions in a chain (taking apart, products, softmax, products), with barriers around the first. What is not finite, and
// scores that overflow, go by multiply-adds over the keys a row sees. Few rows behind long contexts share their keys among the blocks
// of a cluster, which merge through each other's shared memory.
//
// Single tokens: bound by the stream of keys and values. A half-warp takes whole keys (16 lanes x 16 bytes), four in
// flight with their values, for all heads of the group; the keys of a token are shared out over `nsplit` blocks and their
// eight half-warps, each with a softmax of its own, merged in a fixed order in the block, then by a second kernel.
//
// The prompt kernel (us; by multiply-adds, 4 x 4 of them a thread, in brackets): 16 heads over 8 on 1,000 tokens 74 (153), on 300 29 (40), on
// 64 8.3 (9.7), 33 behind 2,500 positions 37 (226), 3 x 700 behind 2,500 586 (890); against 64 bits 1e-7 to 2.5e-7 off (2e-7 to 8e-7).
#include <cooperative_groups.h>
#include <math.h>

#include "paged_tiles.cuh"
#include "parts.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr int F_D = 64, F_ROWS = 64, F_KEYS = 64, F_THREADS = 128;
constexpr int F_PART = F_KEYS * F_D * 2;                  // bytes of one 16-bit part of a tile
constexpr int F_STAGE = F_KEYS * F_D * 4;                 // bytes of a tile of floats
constexpr int F_Q = 6 * F_PART + 2 * F_STAGE;           // q in parts, as the registers hold it: [warp][16 columns][part][lane]
constexpr int F_SMEM = F_Q + 4 * 4 * 3 * 512;

// (high, rest) of four neighbouring tiles += a float's parts times another's, the six largest of the nine products; the operand's
// halves lie at b0 and b1, each in three 16-bit tiles. The same product of all four tiles in a row: a chain's next one waits for nothing.
template <bool TURNED>
__device__ __forceinline__ void six_products(float (&hi)[8][4], float (&lo)[8][4], int n, const uint32_t (&a)[3][4], uint32_t b0, uint32_t b1) {
    uint32_t b[3][2][4];
#pragma unroll
    for (int p = 0; p < 3; ++p) {
        if constexpr (TURNED) {
            ldmatrix_x4_trans(b[p][0], b0 + p * F_PART);
            ldmatrix_x4_trans(b[p][1], b1 + p * F_PART);
        } else {
            ldmatrix_x4(b[p][0], b0 + p * F_PART);
            ldmatrix_x4(b[p][1], b1 + p * F_PART);
        }
    }
    auto all = [&](float (&c)[8][4], int pa, int pb) {
#pragma unroll
        for (int i = 0; i < 4; ++i) mma16816(c[n + i], a[pa], b[pb][i >> 1][(i & 1) * 2], b[pb][i >> 1][(i & 1) * 2 + 1]);
    };
    all(hi, 0, 0);
    all(lo, 2, 0);
    all(lo, 1, 1);
    all(lo, 0, 2);
    all(lo, 1, 0);
    all(lo, 0, 1);
}

// The blocks of a cluster share the keys of their 64 rows, every nsplit-th tile each, as many of them as leave each F_MIN_TILES tiles (the
// others exit); then each merges an equal part of the rows from the others' shared memory.
constexpr int F_MIN_TILES = 3;

__global__ void __launch_bounds__(F_THREADS, 2)
attn32_prefill_kernel(const float* q, const float* kv_pool, float* out, const int* positions, const int* tok_seq,
                      const int* block_table, int bt_stride, const int* tile_tok0, const int* tile_ntok, int H, int Hkv,
                      int P, int window, float scale, int max_split) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ int64_t key_at[2][F_KEYS];    // where a key's row begins in the pool (-1: no such key), of this tile and the next
    const uint32_t kt = (uint32_t)__cvta_generic_to_shared(smem), vt = kt + 3 * F_PART, stage = vt + 3 * F_PART;
    const int G = H / Hkv, split = blockIdx.x % max_split, kvh = blockIdx.x / max_split % Hkv;
    // the longest tiles of a list come last in it: they are begun first
    const int tile = gridDim.x / (Hkv * max_split) - 1 - blockIdx.x / (Hkv * max_split);
    const int tok0 = tile_tok0[tile], ntok = tile_ntok[tile];
    if (ntok <= 0) return;                   // an unused entry of a fixed-length tile list (captured steps)
    const int rows = ntok * G, seq = tok_seq[tok0], tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tok = 2 * (lane & 3);          // the accumulators' first column of eight
    const int lo = first_seen(positions[tok0], window), last = positions[tok0 + ntok - 1];
    const int all_tiles = (last - lo) / F_KEYS + 1, nsplit = min(max_split, max(1, all_tiles / F_MIN_TILES));
    if (split >= nsplit) return;
    const int step = nsplit * F_KEYS;
    const int64_t v_off = (int64_t)Hkv * P * F_D;
    auto find = [&](int j0, int turn) {      // the rows of the tile that begins at j0
        if (tid >= F_KEYS) return;
        const int j = j0 + tid;
        int64_t at = -1;
        if (j <= last) {
            const int page = TK_PAGE(TK_K_ATTN_GENERIC, block_table[(size_t)seq * bt_stride + j / P]);
            at = (((int64_t)page * 2 * Hkv + kvh) * P + j % P) * F_D;
        }
        key_at[turn & 1][tid] = at;
    };
    auto fetch = [&](int j0, int turn) {
        if (j0 <= last) {
            const int64_t* rows_at = key_at[turn & 1];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const int i = tid + e * F_THREADS;
                const int64_t at = rows_at[i >> 4];
                const float* src = kv_pool + (at < 0 ? 0 : at) + (i & 15) * 4;
                cp_async16(stage + i * 16, src, at >= 0);
                cp_async16(stage + F_STAGE + i * 16, at < 0 ? src : src + v_off, at >= 0);
            }
        }
        cp_async_commit();
    };
    const int begin = lo + split * F_KEYS;
    find(begin, 0);
    __syncthreads();
    fetch(begin, 0);

    int pos[2], seen[2];                     // this thread's rows: their position and the first one they see
    const float* q_row[2];
    uint8_t* const q_parts = smem + F_Q + warp * 4 * 3 * 512 + lane * 16;
    float probe = 0.f;                       // stays 0 while every number it has met is finite
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int r = warp * 16 + (lane >> 2) + 8 * i, rr = r < rows ? r : 0;
        pos[i] = r < rows ? positions[tok0 + r / G] : -1;
        seen[i] = first_seen(pos[i], window);
        q_row[i] = q + ((size_t)(tok0 + rr / G) * H + kvh * G + rr % G) * F_D;
    }
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
        uint32_t a[3][4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {        // rows, then rows + 8, of the first eight columns, then of the next
            const float2 v = *reinterpret_cast<const float2*>(q_row[e & 1] + ks * 16 + (e >> 1) * 8 + tok);
            probe = fmaf(v.x, 0.f, fmaf(v.y, 0.f, probe));
            take_apart(v.x, v.y, a[0][e], a[1][e], a[2][e]);
        }
#pragma unroll
        for (int p = 0; p < 3; ++p) *reinterpret_cast<uint4*>(q_parts + (ks * 3 + p) * 512) = make_uint4(a[p][0], a[p][1], a[p][2], a[p][3]);
    }
    const bool working = warp * 16 < rows;
    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
    float o[8][4];
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[n][e] = 0.f;
    const uint32_t b_row = (lane & 7) + (lane >> 4) * 8, b_chunk = (lane >> 3) & 1;

    for (int j0 = begin, turn = 0; j0 <= last; j0 += step, ++turn) {
        cp_async_wait<0>();
        __syncthreads();                     // the tile before is done with
        if (j0 + step <= last) find(j0 + step, turn + 1);
        float bad = probe;
#pragma unroll 4
        for (int e = 0; e < 16; ++e) {       // a thread's own sixteen bytes of keys, then of values
            const int i = tid + (e & 7) * F_THREADS;
            const float4 v = *reinterpret_cast<const float4*>(smem + 6 * F_PART + (e >> 3) * F_STAGE + i * 16);
            bad = fmaf(v.x, 0.f, fmaf(v.y, 0.f, fmaf(v.z, 0.f, fmaf(v.w, 0.f, bad))));
            uint2 part[3];
            cut_apart(v.x, v.y, part[0].x, part[1].x, part[2].x);
            cut_apart(v.z, v.w, part[0].y, part[1].y, part[2].y);
            uint8_t* dst = smem + (e >> 3) * 3 * F_PART + tile_off<F_D>(i >> 4, (i & 15) >> 1) + (i & 1) * 8;
#pragma unroll
            for (int p = 0; p < 3; ++p) *reinterpret_cast<uint2*>(dst + p * F_PART) = part[p];
        }
        const int guarded = __syncthreads_or(bad != 0.f);
        fetch(j0 + step, turn + 1);
        if (!working) continue;
        float s[8][4], overflow = guarded ? 1.f : 0.f;
        if (!guarded) {
            float rest[8][4];
#pragma unroll
            for (int n = 0; n < 8; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) rest[n][e] = 0.f;
#pragma unroll
            for (int part = 0; part < 2; ++part) {
                float hi[8][4];
#pragma unroll
                for (int n = 0; n < 8; ++n)
#pragma unroll
                    for (int e = 0; e < 4; ++e) hi[n][e] = 0.f;
#pragma unroll
                for (int ks = 2 * part; ks < 2 * part + 2; ++ks) {
                    uint32_t a[3][4];
#pragma unroll
                    for (int p = 0; p < 3; ++p) {
                        const uint4 v = *reinterpret_cast<const uint4*>(q_parts + (ks * 3 + p) * 512);
                        a[p][0] = v.x, a[p][1] = v.y, a[p][2] = v.z, a[p][3] = v.w;
                    }
#pragma unroll
                    for (int n = 0; n < 8; n += 4)
                        six_products<false>(hi, rest, n, a, kt + tile_off<F_D>(n * 8 + b_row, ks * 2 + b_chunk),
                                            kt + tile_off<F_D>(n * 8 + 16 + b_row, ks * 2 + b_chunk));
                }
#pragma unroll
                for (int n = 0; n < 8; ++n)
#pragma unroll
                    for (int e = 0; e < 4; ++e) s[n][e] = part == 0 ? hi[n][e] : s[n][e] + hi[n][e];
            }
#pragma unroll
            for (int n = 0; n < 8; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    s[n][e] += rest[n][e];
                    overflow = fmaf(s[n][e], 0.f, overflow);
                }
        }
        if (__any_sync(0xffffffffu, overflow != 0.f)) {
            // something in the tile or in q is not finite, or a product overflows: multiply-adds in the order of d
            const int64_t* rows_at = key_at[turn & 1];
#pragma unroll
            for (int n = 0; n < 8; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int64_t at = rows_at[n * 8 + tok + (e & 1)];
                    float sum = 0.f;
                    if (at >= 0)
#pragma unroll 1
                        for (int d = 0; d < F_D; ++d) sum = fmaf(q_row[e >> 1][d], kv_pool[at + d], sum);
                    s[n][e] = sum;
                }
        }
        float alpha[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            float mx = -INFINITY;
#pragma unroll
            for (int n = 0; n < 8; ++n)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int key = j0 + n * 8 + tok + e;
                    float& v = s[n][2 * i + e];
                    v = key <= pos[i] && key >= seen[i] ? v * scale : -INFINITY;
                    mx = fmaxf(mx, v);
                }
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
            const float m_new = fmaxf(m[i], mx), m_safe = m_new == -INFINITY ? 0.f : m_new;
            alpha[i] = expf(m[i] - m_safe);
            m[i] = m_new;
            float sum = 0.f;
#pragma unroll
            for (int n = 0; n < 8; ++n)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    float& v = s[n][2 * i + e];
                    v = expf(v - m_safe);
                    sum += v;
                }
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            sum += __shfl_xor_sync(0xffffffffu, sum, 2);
            l[i] = l[i] * alpha[i] + sum;
        }
        if (!guarded) {
#pragma unroll
            for (int part = 0; part < 2; ++part) {       // 32 keys at a time: the shorter chain, the less the tensor cores cut off
                float hi[8][4], rest[8][4];
#pragma unroll
                for (int n = 0; n < 8; ++n)
#pragma unroll
                    for (int e = 0; e < 4; ++e) hi[n][e] = rest[n][e] = 0.f;
#pragma unroll
                for (int ks = 2 * part; ks < 2 * part + 2; ++ks) {
                    uint32_t a[3][4];
                    take_apart(s[2 * ks][0], s[2 * ks][1], a[0][0], a[1][0], a[2][0]);
                    take_apart(s[2 * ks][2], s[2 * ks][3], a[0][1], a[1][1], a[2][1]);
                    take_apart(s[2 * ks + 1][0], s[2 * ks + 1][1], a[0][2], a[1][2], a[2][2]);
                    take_apart(s[2 * ks + 1][2], s[2 * ks + 1][3], a[0][3], a[1][3], a[2][3]);
#pragma unroll
                    for (int n = 0; n < 8; n += 4)
                        six_products<true>(hi, rest, n, a, vt + tile_off<F_D>(ks * 16 + (lane & 15), n + (lane >> 4)),
                                           vt + tile_off<F_D>(ks * 16 + (lane & 15), n + 2 + (lane >> 4)));
                }
#pragma unroll
                for (int n = 0; n < 8; ++n)
#pragma unroll
                    for (int e = 0; e < 4; ++e) o[n][e] = fmaf(part == 0 ? alpha[e >> 1] : 1.f, o[n][e], hi[n][e] + rest[n][e]);
            }
            continue;
        }
        // a weight of zero does not hide a value that is not finite: the keys a row sees, and no others
        const int64_t* rows_at = key_at[turn & 1];
#pragma unroll
        for (int n = 0; n < 8; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) o[n][e] *= alpha[e >> 1];
#pragma unroll
        for (int n = 0; n < 8; ++n)
#pragma unroll 1
            for (int k = 0; k < 8; ++k) {
                const int from = (lane & ~3) | (k >> 1), key = j0 + n * 8 + k;
                const float p0 = __shfl_sync(0xffffffffu, k & 1 ? s[n][1] : s[n][0], from);
                const float p1 = __shfl_sync(0xffffffffu, k & 1 ? s[n][3] : s[n][2], from);
                const int64_t at = rows_at[n * 8 + k];
                if (at < 0) continue;
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const float2 v = *reinterpret_cast<const float2*>(kv_pool + at + v_off + c * 8 + tok);
                    if (key <= pos[0] && key >= seen[0]) o[c][0] = fmaf(p0, v.x, o[c][0]), o[c][1] = fmaf(p0, v.y, o[c][1]);
                    if (key <= pos[1] && key >= seen[1]) o[c][2] = fmaf(p1, v.x, o[c][2]), o[c][3] = fmaf(p1, v.y, o[c][3]);
                }
            }
    }
    pdl_launch_dependents();                 // (not earlier: see the launch)
    cp_async_wait<0>();
    if (nsplit == 1) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int r = warp * 16 + (lane >> 2) + 8 * i;
            if (r >= rows) continue;
            float* dst = out + ((size_t)(tok0 + r / G) * H + kvh * G + r % G) * F_D + tok;
            const float inv = l[i] > 0.f ? 1.0f / l[i] : 0.f;
#pragma unroll
            for (int n = 0; n < 8; ++n) *reinterpret_cast<float2*>(dst + n * 8) = make_float2(o[n][2 * i] * inv, o[n][2 * i + 1] * inv);
        }
        return;
    }
    __syncthreads();                         // the tiles are done with: this block's rows in their place, then their maxima and sums
    float* o_s = reinterpret_cast<float*>(smem);
    float2* ml_s = reinterpret_cast<float2*>(smem + F_ROWS * F_D * 4);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int r = warp * 16 + (lane >> 2) + 8 * i;
#pragma unroll
        for (int n = 0; n < 8; ++n) *reinterpret_cast<float2*>(o_s + r * F_D + n * 8 + tok) = make_float2(o[n][2 * i], o[n][2 * i + 1]);
        if (tok == 0) ml_s[r] = make_float2(m[i], l[i]);
    }
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    // 16 lanes a row, four columns each
    for (int r = split * (F_THREADS / 16) + (tid >> 4); r < rows; r += nsplit * (F_THREADS / 16)) {
        float M = -INFINITY, L = 0.f;
        for (int sp = 0; sp < nsplit; ++sp) M = fmaxf(M, cluster.map_shared_rank(ml_s, sp)[r].x);
        float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int sp = 0; sp < nsplit; ++sp) {
            const float2 one = cluster.map_shared_rank(ml_s, sp)[r];
            const float f = one.x == -INFINITY ? 0.f : expf(one.x - M);
            const float4 v = *reinterpret_cast<const float4*>(cluster.map_shared_rank(o_s, sp) + r * F_D + (tid & 15) * 4);
            L = fmaf(one.y, f, L);
            sum.x = fmaf(v.x, f, sum.x), sum.y = fmaf(v.y, f, sum.y), sum.z = fmaf(v.z, f, sum.z), sum.w = fmaf(v.w, f, sum.w);
        }
        const float inv = L > 0.f ? 1.0f / L : 0.f;
        *reinterpret_cast<float4*>(out + ((size_t)(tok0 + r / G) * H + kvh * G + r % G) * F_D + (tid & 15) * 4) =
            make_float4(sum.x * inv, sum.y * inv, sum.z * inv, sum.w * inv);
    }
    cluster.sync();                          // nobody leaves while its rows are read
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
// sequence with consecutive positions; window: see first_seen. nsplit (1, 2, 4 or 8): up to that many blocks share a tile's keys.
TK_API int tk_attn_f32_prefill(const void* q, const void* kv_pool, void* out, const int* positions, const int* tok_seq,
                               const int* block_table, int bt_stride, const int* tile_tok0, const int* tile_ntok, int n_tiles,
                               int H, int Hkv, int P, int window, float scale, int nsplit, cudaStream_t stream) {
    TK_CHECK_ARG(tk_attn_f32_supported(H, Hkv, F_D), "attention (32-bit): %d query heads over %d KV heads", H, Hkv);
    TK_CHECK_ARG(nsplit == 1 || nsplit == 2 || nsplit == 4 || nsplit == 8, "attention (32-bit): %d splits (1, 2, 4 or 8)", nsplit);
    TK_CHECK_ARG(P > 0 && n_tiles >= 0 && (int64_t)n_tiles * Hkv * nsplit < 0x7fffffff, "attention (32-bit): bad page size or tile count");
    TK_CHECK_ARG((uintptr_t)q % 16 == 0 && (uintptr_t)kv_pool % 16 == 0, "attention (32-bit): 16-byte aligned bases");
    if (n_tiles == 0) return 0;
    cudaFuncSetAttribute(attn32_prefill_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, F_SMEM);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(n_tiles * Hkv * nsplit);
    cfg.blockDim = dim3(F_THREADS);
    cfg.dynamicSmemBytes = F_SMEM;
    cfg.stream = stream;
    // In plain stream order, and its dependents are let in at its end: blocks of 104 KB that come while the product before still runs, and the
    // next product's that come among these, lie several to one SM and none to another for their whole run (layers of 16 heads over 8:
    // 64 tokens 37.5 us, 40.1 otherwise, 37.9 with the kernel before this one, whose blocks were smaller; of 32 heads, 512 tokens 163.6,
    // 172.8 and 174.4, eight prompts of 64 118.9, 127.8 and 121.5).
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = nsplit;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = nsplit > 1 ? 1 : 0;
    cudaLaunchKernelEx(&cfg, attn32_prefill_kernel, (const float*)q, (const float*)kv_pool, (float*)out, positions, tok_seq, block_table,
                       bt_stride, tile_tok0, tile_ntok, H, Hkv, P, window, scale, nsplit);
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
