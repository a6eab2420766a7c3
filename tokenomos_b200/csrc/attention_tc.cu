// Paged prefill attention on the fifth-generation tensor cores, for bfloat16 and head size 64:
// S = Q K^T and O += P V are tcgen05.mma instructions with their accumulators in tensor memory;
// the online softmax runs on 2 x 128 threads, one query row of one key tile each.
//
// A CTA takes up to 128 rows: 128 / G tokens of one sequence with the G query heads that share one
// KV head (row = token * G + head), and walks the keys in tiles of 64, this step's own keys
// included. Warps coupled by mbarriers only:
//
//   warp 0      brings K and V from the paged cache by TMA, a page (or 64 rows of one) a load, into
//               128-byte-swizzled tiles, up to six tiles ahead; rows of a ragged tile that nobody may
//               read are zeroed after they land. Both are used as they land: K's [key][d] is the K-major B operand of
//               S = Q K^T, V's the MN-major B operand of P V. (Pages of less than 8 positions, or not a
//               power of two: warps 0-1 by cp.async.)
//   warp 3      one lane issues the MMAs: S_j (128 x 64 x 64), and P_j V_j into one of two outputs
//               that live in tensor memory for the whole walk.
//   warps 4-11  bring Q, then are two groups of 128 threads that take the key tiles in turn, each with scores, weights
//               and an output of its own, so that one's chain (scores from tensor memory, maximum,
//               exponentials, weights, the two products) runs under the other's. Thread r owns row
//               r of its group's tiles: masks (causal, window), keeps a reference maximum and the row
//               sum in 32-bit, and writes P_j as bfloat16 into the tensor memory that S_j held, where
//               the second product reads it as its A operand. The reference maximum
//               follows the true one lazily (see the softmax section); only when it is raised is
//               the accumulated output read, scaled and written back (tcgen05.ld / tcgen05.st). At the
//               end the first group reads both outputs (a warp's lanes of tensor memory are the same
//               in both) and merges them.
//
// Bound by each group's chain: 2,500 cycles a tile alone on an SM (scores there 100, maximum 330, exponentials 850, the
// products' issue and the barriers around them 1,200), 3,000 beside a second CTA, where four chains keep the special-function
// unit (512 cycles a tile) at two thirds. One group of 128 threads a CTA, with V turned by ldmatrix and stmatrix, took
// 2,700 a tile and CTA: 512 tokens of 32 heads over 8 behind 8,192 positions 89 us, now 70; a prompt of 2,048 48.3 and 39.8; 3 x 700
// behind 2,500 (the layer) 190 and 141; 128 tokens of 16 heads behind 32,000, whose keys 16 CTAs shared and now 8, 60
// and 68. At 80 registers a thread the compiler spills 140 bytes of a thread (3 % of the instructions it runs).
//
// Masking, scale, rounding of P to bfloat16 and the unrounded row sum are those of the other
// attention kernels (Tokenomos kernels/attention/paged.py:67-76,150,267;
// models/blocks/attention.py:31-40,173). Rows of a page beside the positions a tile sees come with it and are
// zeroed before a product reads them.
//
// Every mbarrier wait is bounded (about a second, or until another thread has recorded an
// error); the kernel then leaves its loops, frees its tensor memory and returns, and
// tk_attn_prefill_tc_status() reports where it gave up.
#include <cooperative_groups.h>
#include <math.h>

#include <type_traits>

#include "paged_tiles.cuh"
#include "tcgen05.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr int AT_D = 64;                  // head size
constexpr int AT_ROWS = 128;              // query rows per CTA (UMMA M)
constexpr int AT_KEYS = 64;               // keys per tile (UMMA N of S, K of P V)
constexpr int AT_THREADS = 384;           // TMA warp (or two that copy), MMA warp, 2 x 4 softmax warps
constexpr int AT_STAGING = 64;            // threads that copy
constexpr int AT_STAGES = 6;              // key / value tiles in shared memory
constexpr int AT_KV_BYTES = AT_KEYS * AT_D * 2;
constexpr int AT_Q_BYTES = AT_ROWS * AT_D * 2;
// dynamic shared memory: Q, K and V stages, barriers; two blocks fit an SM
constexpr int AT_SMEM = AT_Q_BYTES + 2 * AT_STAGES * AT_KV_BYTES + 256;
constexpr int AT_SHARE_LD = AT_D + 4;
constexpr int AT_SPLIT_TILES = 8;         // key tiles a CTA should have before a tile's keys are shared out
constexpr float AT_LAZY = 8.0f;           // log2 of how far a probability may exceed 1 before a rescale
constexpr long long AT_WAIT_CYCLES = 2000000000LL;

__device__ int g_at_error = 0;

__device__ __forceinline__ bool at_wait(uint32_t bar, uint32_t parity, int where) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long start = clock64();
    int it = 0;
    while (!mbar_try_wait(bar, parity)) {
        if ((++it & 255) == 0) {
            if (*(volatile int*)&g_at_error != 0) return false;
            if (clock64() - start > AT_WAIT_CYCLES) {
                atomicCAS(&g_at_error, 0, where);
                return false;
            }
        }
    }
    return true;
}

// True in one lane of a converged warp, the same one every time.
__device__ __forceinline__ bool elect_lane() {
    uint32_t mine;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(mine));
    return mine != 0;
}

// D += A B with A (bfloat16, two to a 32-bit column) in tensor memory
__device__ __forceinline__ void umma_bf16_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ uint32_t pack_bf16_pair(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}

// Packed 32-bit arithmetic (two lanes per instruction): the softmax threads are bound by the
// number of instructions they issue, and most of them are elementwise on pairs.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }

__device__ __forceinline__ float fmax3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// Options of a layer's attention beyond window and scale (X = true compiles them in; the plain
// kernel is the X = false one). `keep_first`: with a window, keys at positions below it stay
// visible to every later query: their key tiles come first in a CTA's list, then the window's.
// `sink`: the softmax's denominator has one more term, a key of score 0 without a value: the
// reference maximum and the row sum start from it (in the first of a tile's shares only).
// `gate_mode` 2: the gate has one value per output element ([T, H * 64] rows `ldg` apart), and the
// 32-bit output times the 32-bit sigmoid is rounded once.
struct AtOptions {
    int keep_first;
    int sink;
    int gate_mode;
};

template <bool X>
__global__ void __launch_bounds__(AT_THREADS, 2)
attn_prefill_tc_kernel(const __nv_bfloat16* q, const __nv_bfloat16* pool, __nv_bfloat16* out,
                       const int* positions, const int* tok_seq, const int* block_table, int bt_stride,
                       const int* tile_tok0, const int* tile_ntok, int H, int Hkv, int P, int window,
                       float scale, int p_shift, const __grid_constant__ CUtensorMap kv_map, const __nv_bfloat16* gate, int64_t ldg, int max_split,
                       const AtOptions opt) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    pdl_launch_dependents();
    if (threadIdx.x == 0 && p_shift >= 3)            // (the map is the launch's own: fetched while the kernel before ends)
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&kv_map)) : "memory");
    pdl_wait();
    // (no static shared memory: the dynamic part begins on 1,024 bytes, as the swizzled tiles must)
    const uint32_t base = smem_u32(smem_raw);
    if ((base & 1023u) != 0) {
        if (threadIdx.x == 0) atomicCAS(&g_at_error, 0, 9);
        return;
    }
    const uint32_t q_tile = base;
    const uint32_t k_tile0 = q_tile + AT_Q_BYTES;                         // AT_STAGES stages
    const uint32_t v_tile0 = k_tile0 + AT_STAGES * AT_KV_BYTES;           // [key][d], as it lands
    const uint32_t bars = v_tile0 + AT_STAGES * AT_KV_BYTES;
    auto kv_full = [&](int s) { return bars + (uint32_t)s * 8; };
    auto kv_empty = [&](int s) { return bars + (uint32_t)(AT_STAGES + s) * 8; };
    auto s_full = [&](int b) { return bars + (uint32_t)(2 * AT_STAGES + b) * 8; };
    auto p_full = [&](int b) { return bars + (uint32_t)(2 * AT_STAGES + 2 + b) * 8; };
    auto pv_full = [&](int b) { return bars + (uint32_t)(2 * AT_STAGES + 4 + b) * 8; };
    const uint32_t q_full = bars + (2 * AT_STAGES + 6) * 8, ragged = q_full + 8;
    const uint32_t tmem_slot = ragged + 8;
    volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(smem_raw + (tmem_slot - base));

    // a share of the keys, when several CTAs have one: rows 68 floats apart, then each row's maximum and sum
    float* share_o = reinterpret_cast<float*>(smem_raw + AT_Q_BYTES);
    float2* share_ml = reinterpret_cast<float2*>(share_o + AT_ROWS * AT_SHARE_LD);

    const int G = H / Hkv;
    // the grid is one-dimensional with the KV head fastest and the tiles in reverse: a causal
    // tile late in its sequence reads the most keys, so the longest CTAs start first
    const int group = blockIdx.x / max_split, kvh = group % Hkv;
    const int tile = gridDim.x / (max_split * Hkv) - 1 - group / Hkv;
    const int tok0 = tile_tok0[tile], ntok = tile_ntok[tile];
    if (ntok <= 0) return;       // an unused entry of a fixed-length tile list (captured steps)
    const int rows = ntok * G;
    const int seq = tok_seq[tok0];
    const int* bt_row = block_table + (size_t)seq * bt_stride;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int pos_first = positions[tok0];
    const int pos_last = pos_first + ntok - 1;       // consecutive positions within a tile
    const int lo = first_seen(pos_first, window);
    const int j_begin = (lo / AT_KEYS) * AT_KEYS;
    // Up to `max_split` CTAs, a cluster, share a tile's keys, as many as leave each at least
    // AT_SPLIT_TILES key tiles: CTA `split` takes key tiles split, split + nsplit, ...; the ones
    // beyond that number have nothing to do. (The launch fixes the most; the tile decides.)
    const int split = blockIdx.x % max_split;
    // the kept positions that lie before the window of the tile's first row, [0, keep_end), come
    // first in the list of key tiles
    const int keep_first = X ? opt.keep_first : 0;
    const int keep_end = (keep_first > 0 && lo > 0) ? min(keep_first, lo) : 0;
    const int n_keep = (keep_end + AT_KEYS - 1) / AT_KEYS;
    const int all_tiles = n_keep + (pos_last - j_begin) / AT_KEYS + 1;
    const int most = min(max_split, max(1, all_tiles / AT_SPLIT_TILES)), nsplit = most >= 8 ? 8 : most >= 4 ? 4 : most >= 2 ? 2 : 1;
    if (split >= nsplit) return;
    const int n_tiles = (all_tiles - split + nsplit - 1) / nsplit;       // at least one
    // key tile `it` of this CTA: its first key, and the first and last key it may read
    auto tile_j0 = [&](int it) {
        const int t = split + it * nsplit;
        return t < n_keep ? t * AT_KEYS : j_begin + (t - n_keep) * AT_KEYS;
    };
    auto tile_lo = [&](int it) { return split + it * nsplit < n_keep ? 0 : lo; };
    auto tile_hi = [&](int it) { return split + it * nsplit < n_keep ? keep_end - 1 : pos_last; };

    if (tid == 0) {
        for (int i = 0; i < AT_STAGES; ++i) {
            mbar_init(kv_full(i), 1);
            mbar_init(kv_empty(i), 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(s_full(i), 1);
            mbar_init(p_full(i), 4);
            mbar_init(pv_full(i), 1);
        }
        mbar_init(q_full, 8);
        mbar_init(ragged, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 3) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(256u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot_ptr;
    const uint32_t tmem_pv = tmem + 2 * AT_KEYS;         // outputs at columns 128 + 64 b; S_b at [64 b, 64 b + 64)

    // The register file is shared unevenly: the first four warps give registers up and the softmax
    // warps (a whole row of scores each) take them: 128 x 48 + 256 x 96 of the launch's 384 x 80.
    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 48;");
        const bool by_pages = p_shift >= 3;
        if (warp == 0 && by_pages) {
            // ---- K and V by TMA ----
            bool ok = true;
            const int per_log = min(p_shift, 6), per = 1 << per_log;         // rows of a load
            int n_ragged = 0;
            for (int it = 0; it < n_tiles && ok; ++it) {
                const int s = it % AT_STAGES, j0 = tile_j0(it), first = tile_lo(it), last = tile_hi(it);
                const uint32_t kt = k_tile0 + (uint32_t)s * AT_KV_BYTES, vt = v_tile0 + (uint32_t)s * AT_KV_BYTES;
                // lane l brings rows [l per, (l + 1) per) of the tile, if any of them may be read
                const int jl = j0 + lane * per;
                const bool mine = lane < (AT_KEYS >> per_log) && jl <= last && jl + per > first;
                int page = 0;
                if (mine) page = TK_PAGE(TK_K_ATTN_TILES, bt_row[jl >> p_shift]);
                if (it >= AT_STAGES) ok = at_wait(kv_empty(s), (uint32_t)((it / AT_STAGES - 1) & 1), 1);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                const bool whole = j0 >= first && j0 + AT_KEYS - 1 <= last;
                const uint32_t bar = whole ? kv_full(s) : ragged;
                const int loads = __popc(__ballot_sync(0xffffffffu, mine));
                if (lane == 0) mbar_expect_tx(bar, (uint32_t)(loads * 2 * per * AT_D * 2));
                __syncwarp();
                if (mine) {
                    const int row = ((page * 2) * Hkv + kvh) * P + (jl & (P - 1));
                    tma_load_2d(kt + (uint32_t)(lane * per) * (AT_D * 2), &kv_map, 0, row, bar);
                    tma_load_2d(vt + (uint32_t)(lane * per) * (AT_D * 2), &kv_map, 0, row + Hkv * P, bar);
                }
                if (whole) continue;
                // a ragged tile: what nobody may read is zeroed, whatever the cache holds there
                ok = at_wait(ragged, (uint32_t)(n_ragged++ & 1), 10);
                ok = __all_sync(0xffffffffu, ok);
                for (int i = lane; i < AT_KEYS * 8; i += 32) {
                    const int j = j0 + (i >> 3);
                    if (j >= first && j <= last) continue;
                    const uint32_t at = (uint32_t)i * 16;
                    asm volatile("st.shared.v4.b32 [%0], {%1,%1,%1,%1};" ::"r"(kt + at), "r"(0) : "memory");
                    asm volatile("st.shared.v4.b32 [%0], {%1,%1,%1,%1};" ::"r"(vt + at), "r"(0) : "memory");
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(kv_full(s));
            }
        } else if (warp < 2 && !by_pages) {
            // two copies in flight when a tile is handed over
            bool ok = true;
            auto issue = [&](int it) {
                if (it < n_tiles) {
                    const int s = it % AT_STAGES;
                    if (it >= AT_STAGES && ok) ok = at_wait(kv_empty(s), (uint32_t)((it / AT_STAGES - 1) & 1), 1);
                    for (int which = 0; which < 2; ++which)
                        load_tile<AT_D>((which ? v_tile0 : k_tile0) + (uint32_t)s * AT_KV_BYTES, pool, bt_row, tile_j0(it), AT_KEYS,
                                        tile_lo(it), tile_hi(it), kvh, Hkv, P, which, tid, AT_STAGING);
                }
                cp_async_commit();
            };
            issue(0);
            issue(1);
            // (after a failed wait the loop still runs to its end, without waiting: every thread must
            // meet every named barrier)
            for (int it = 0; it < n_tiles; ++it) {
                cp_async_wait<1>();
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                asm volatile("bar.sync 2, 64;" ::: "memory");
                if (tid == 0) mbar_arrive(kv_full(it % AT_STAGES));
                issue(it + 2);
            }
            cp_async_wait<0>();
        } else if (warp == 3) {
            // ---- MMA issuer: the warp walks the tiles together, so that descriptors and addresses are formed in uniform
            // registers (one lane alone takes 850 cycles a tile to hand them over), one elected lane issues ----
            constexpr uint32_t idesc = umma_idesc(AT_KEYS);      // 128 x 64
            constexpr uint32_t idesc_pv = idesc | (1u << 16);    // the same, B as [key][d]: MN-major
            const uint64_t qdesc = umma_desc(q_tile);
            auto wait = [&](uint32_t bar, uint32_t parity, int where) { return __all_sync(0xffffffffu, at_wait(bar, parity, where)) != 0; };
            bool ok = wait(q_full, 0, 3);
            auto issue_s = [&](int j) {
                const int s = j % AT_STAGES, b = j & 1;
                ok = ok && wait(kv_full(s), (uint32_t)((j / AT_STAGES) & 1), 2);
                if (!ok) return;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t kdesc = umma_desc(k_tile0 + (uint32_t)s * AT_KV_BYTES);
                if (elect_lane()) {
#pragma unroll
                    for (int k = 0; k < AT_D / 16; ++k)
                        umma_bf16(tmem + (uint32_t)b * AT_KEYS, qdesc + 2 * k, kdesc + 2 * k, idesc, k > 0 ? 1u : 0u);
                    umma_commit(s_full(b));
                }
                __syncwarp();
            };
            issue_s(0);
            if (n_tiles > 1) issue_s(1);
            for (int j = 0; j < n_tiles && ok; ++j) {
                const int s = j % AT_STAGES, b = j & 1;
                ok = wait(p_full(b), (uint32_t)((j >> 1) & 1), 4);    // P_j written, the output rescaled if need be
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t vdesc = umma_desc(v_tile0 + (uint32_t)s * AT_KV_BYTES);
                if (elect_lane()) {
#pragma unroll
                    for (int k = 0; k < AT_KEYS / 16; ++k)           // 16 keys: 8 columns of P, 16 rows of V
                        umma_bf16_ta(tmem_pv + (uint32_t)b * AT_D, tmem + (uint32_t)(b * AT_KEYS + 8 * k), vdesc + 128 * k, idesc_pv,
                                     (j > 1 || k > 0) ? 1u : 0u);
                }
                __syncwarp();
                // (in order behind the product that reads P_j, where S_{j+2} goes; the group's next wait is for it, and for that product)
                if (j + 2 < n_tiles) issue_s(j + 2);
                // (one phase of pv_full: a group that skipped phases could not tell by a phase's one bit which is open)
                if (elect_lane()) {
                    if (j + 2 >= n_tiles) umma_commit(pv_full(b));
                    umma_commit(kv_empty(s));
                }
                __syncwarp();
            }
        }
        __syncwarp();
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 96;");
        // ---- Q: row r = token * G + head (G divides 128: a power of two); rows past the tile are zero ----
        const int g_shift = __ffs(G) - 1;
#pragma unroll
        for (int i = tid - 128; i < AT_ROWS * (AT_D / 8); i += 256) {
            const int rr = i >> 3, c = i & 7;
            const bool valid = rr < rows;
            const __nv_bfloat16* src = q;
            if (valid) src = q + ((size_t)(tok0 + (rr >> g_shift)) * H + kvh * G + (rr & (G - 1))) * AT_D + c * 8;
            cp_async16(q_tile + tile_off<AT_D>(rr, c), src, valid);
        }
        cp_async_commit();
        cp_async_wait<0>();
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(q_full);
        // ---- softmax: thread r of a group owns query row r of the group's key tiles ----
        // The output accumulates in tensor memory over all key tiles (P V with the accumulate
        // flag) under a reference maximum m_ref that follows the true maximum lazily: it is
        // raised, and the accumulated row and sum rescaled, only when some row of the warp sees a
        // score more than AT_LAZY (in log2 units) above it. Until then probabilities may exceed 1,
        // by at most 2^AT_LAZY; in 32-bit accumulation, with the division by the row sum at the
        // end, that changes nothing but the scale the intermediate values live at.
        const int grp = (warp - 4) >> 2, r = (tid - 128) & 127;
        const int quarter = warp & 3;
        const uint32_t out_addr = tmem_pv + (uint32_t)grp * AT_D + ((uint32_t)(quarter * 32) << 16);
        const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
        const int pos_r = r < rows ? pos_first + (r >> g_shift) : -1;
        const int lo_r = first_seen(pos_r, window), lo_last = first_seen(pos_last, window);
        const float scale_log2 = scale * LOG2E;
        float m_ref = -INFINITY;
        float2 l_run = make_float2(0.f, 0.f), l_alt = make_float2(0.f, 0.f);   // the row sum in four lanes
        if (X && opt.sink && split == 0 && grp == 0) {
            m_ref = 0.f;
            l_run.x = 1.f;
        }
        bool ok = true;
        for (int j = grp; j < n_tiles; j += 2) {
            const int b = grp, turn = j >> 1, j0 = tile_j0(j);
            // (after a failed wait the loop still runs to its end, without waiting: every thread
            // must meet the barrier behind it)
            if (ok) ok = at_wait(s_full(b), (uint32_t)(turn & 1), 6);
            ok = __all_sync(0xffffffffu, ok);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t s_addr = tmem + lane_base + (uint32_t)b * AT_KEYS;
            float s_lo[32], s_hi[32];                    // the row's 64 scores stay in registers
            tmem_ld32(s_addr, s_lo);
            tmem_ld32(s_addr + 32u, s_hi);
            // a tile every row of the CTA sees whole needs no comparisons
            const bool kept = X && split + j * nsplit < n_keep;
            // (a row past the tile's rows is a query of zeros whose sums nobody reads)
            const bool masked = j0 + AT_KEYS - 1 > pos_first || j0 < lo_last || kept;
            // what this row sees of the tile: [see_lo, see_hi], and below keep_first whatever the window
            const int see_hi = X ? min(pos_r, tile_hi(j)) : pos_r;
            const int see_lo = X ? tile_lo(j) : 0;
            auto sees = [&](int key) {
                if constexpr (X) return key <= see_hi && key >= see_lo && (key >= lo_r || key < keep_first);
                else return key <= pos_r && key >= lo_r;
            };
            // the row's maximum over the tile's visible keys (the scale is positive)
            // (four chains: a thread has few other warps to hide a 64-deep dependency behind)
            float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
            if (masked) {
#pragma unroll
                for (int e = 0; e < 32; ++e) {
                    const int key = j0 + e;
                    if (sees(key)) mx4[e & 1] = fmaxf(mx4[e & 1], s_lo[e]);
                    if (sees(key + 32)) mx4[2 + (e & 1)] = fmaxf(mx4[2 + (e & 1)], s_hi[e]);
                }
            } else {
#pragma unroll
                for (int e = 0; e < 32; ++e) mx4[e & 3] = fmax3(mx4[e & 3], s_lo[e], s_hi[e]);
            }
            const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * scale_log2;
            const bool raise = __any_sync(0xffffffffu, mx > m_ref + AT_LAZY);
            if (raise) {
                const float m_new = fmaxf(m_ref, mx);
                if (X && turn == 0) {         // nothing accumulated yet but, with a sink, the sum's first term
                    const float alpha0 = m_new == -INFINITY ? 1.0f : fast_exp2(m_ref - m_new);
                    l_run.x *= alpha0;
                }
                if (turn >= 1) {
                    // (the product of the group's tile before has landed: it was issued ahead of these scores, whose commit covers both)
                    const float alpha = m_new == -INFINITY ? 1.0f : fast_exp2(m_ref - m_new);
#pragma unroll
                    for (int c = 0; c < AT_D; c += 16) {          // (narrow: the scores stay in registers)
                        float part[16];
                        tmem_ld16(out_addr + (uint32_t)c, part);
#pragma unroll
                        for (int e = 0; e < 16; ++e) part[e] *= alpha;
                        tmem_st16(out_addr + (uint32_t)c, part);
                    }
                    l_run.x *= alpha;
                    l_run.y *= alpha;
                    l_alt.x *= alpha;
                    l_alt.y *= alpha;
                }
                m_ref = m_new;
            }
            const float neg_m = m_ref == -INFINITY ? 0.f : -m_ref;
            // probabilities, rounded to bfloat16, go where the scores were: the A operand of P V
            auto emit = [&](const float (&part)[32], int c) {
                uint32_t packed[16];
                if (masked) {
#pragma unroll
                    for (int e = 0; e < 32; e += 2) {
                        float p0 = 0.f, p1 = 0.f;
                        const int key = j0 + c + e;
                        if (sees(key)) p0 = fast_exp2(fmaf(part[e], scale_log2, neg_m));
                        if (sees(key + 1)) p1 = fast_exp2(fmaf(part[e + 1], scale_log2, neg_m));
                        if (e & 2) l_alt = add2(l_alt, make_float2(p0, p1));
                        else l_run = add2(l_run, make_float2(p0, p1));
                        packed[e >> 1] = pack_bf16_pair(p0, p1);
                    }
                } else {
                    const float2 sc2 = make_float2(scale_log2, scale_log2), nm2 = make_float2(neg_m, neg_m);
#pragma unroll
                    for (int e = 0; e < 32; e += 2) {
                        const float2 x = fma2(make_float2(part[e], part[e + 1]), sc2, nm2);
                        const float2 pp = make_float2(fast_exp2(x.x), fast_exp2(x.y));
                        if (e & 2) l_alt = add2(l_alt, pp);
                        else l_run = add2(l_run, pp);
                        packed[e >> 1] = pack_bf16_pair(pp.x, pp.y);
                    }
                }
                asm volatile(
                    "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
                    ::"r"(s_addr + (uint32_t)(c >> 1)), "r"(packed[0]), "r"(packed[1]), "r"(packed[2]), "r"(packed[3]), "r"(packed[4]),
                      "r"(packed[5]), "r"(packed[6]), "r"(packed[7]), "r"(packed[8]), "r"(packed[9]), "r"(packed[10]), "r"(packed[11]),
                      "r"(packed[12]), "r"(packed[13]), "r"(packed[14]), "r"(packed[15])
                    : "memory");
            };
            emit(s_lo, 0);
            emit(s_hi, 32);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(p_full(b));
        }
        if (ok && n_tiles > grp) {
            ok = at_wait(pv_full(grp), 0, 8);
            ok = __all_sync(0xffffffffu, ok);
        }
        // The second group's maximum and sum of each row go to Q's tile, which no product reads any more: the last S of either group
        // was issued before the P V waited for above.
        float l_row = (l_run.x + l_run.y) + (l_alt.x + l_alt.y);
        float2* other = reinterpret_cast<float2*>(smem_raw) + r;
        if (grp == 1 && n_tiles > 1) *other = make_float2(m_ref, l_row);
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        asm volatile("bar.sync 5, 256;" ::: "memory");
        if (ok && grp == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            // both outputs under one reference: o = f0 o0 + f1 o1
            const bool two = n_tiles > 1;
            const float2 theirs = two ? *other : make_float2(-INFINITY, 0.f);
            const float m_all = fmaxf(m_ref, theirs.x);
            const float f0 = m_ref == -INFINITY ? 0.f : fast_exp2(m_ref - m_all);
            const float f1 = theirs.x == -INFINITY ? 0.f : fast_exp2(theirs.x - m_all);
            if (two) l_row = fmaf(l_row, f0, theirs.y * f1);
            m_ref = m_all;
            auto read16 = [&](int c, float (&part)[16]) {
                tmem_ld16(out_addr + (uint32_t)c, part);
                float more[16];
                if (two) tmem_ld16(out_addr + (uint32_t)(AT_D + c), more);
#pragma unroll
                for (int e = 0; e < 16; ++e) part[e] = two ? fmaf(part[e], f0, more[e] * f1) : part[e];
            };
            __nv_bfloat16* dst = r < rows ? out + ((size_t)(tok0 + r / G) * H + kvh * G + r % G) * AT_D : nullptr;
            // the per-head output gate, if the layer has one: round(round(o) * round(sigmoid(g)))
            float gs = 1.0f;
            const bool by_element = X && opt.gate_mode == 2;
            const __nv_bfloat16* grow = by_element && dst != nullptr
                                            ? gate + (size_t)(tok0 + r / G) * ldg + (size_t)(kvh * G + r % G) * AT_D
                                            : nullptr;
            if (gate != nullptr && dst != nullptr && !by_element) {
                const float gv = __bfloat162float(gate[(size_t)(tok0 + r / G) * ldg + kvh * G + r % G]);
                gs = round_as<__nv_bfloat16>(1.0f / (1.0f + expf(-gv)));
            }
            // 16 finished values of the row: normalised, rounded, gated, stored
            auto store16 = [&](int c, const float (&part)[16], float inv) {
                if (dst == nullptr) return;
                uint32_t packed[8];
                if (by_element) {
                    const uint4 g0 = *reinterpret_cast<const uint4*>(grow + c), g1 = *reinterpret_cast<const uint4*>(grow + c + 8);
                    const uint32_t gw[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
#pragma unroll
                    for (int e = 0; e < 16; e += 2) {
                        const float2 gv = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&gw[e >> 1]));
                        packed[e >> 1] = pack_bf16_pair(part[e] * inv / (1.0f + __expf(-gv.x)),
                                                        part[e + 1] * inv / (1.0f + __expf(-gv.y)));
                    }
                    *reinterpret_cast<uint4*>(dst + c) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
                    *reinterpret_cast<uint4*>(dst + c + 8) = make_uint4(packed[4], packed[5], packed[6], packed[7]);
                    return;
                }
#pragma unroll
                for (int e = 0; e < 16; e += 2) {
                    packed[e >> 1] = pack_bf16_pair(part[e] * inv, part[e + 1] * inv);
                    if (gate != nullptr) {
                        const float2 f = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&packed[e >> 1]));
                        packed[e >> 1] = pack_bf16_pair(f.x * gs, f.y * gs);
                    }
                }
                *reinterpret_cast<uint4*>(dst + c) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
                *reinterpret_cast<uint4*>(dst + c + 8) = make_uint4(packed[4], packed[5], packed[6], packed[7]);
            };
            if (nsplit == 1) {
                const float inv = l_row > 0.f ? 1.0f / l_row : 0.f;
#pragma unroll
                for (int c = 0; c < AT_D; c += 16) {
                    float part[16];
                    read16(c, part);
                    store16(c, part, inv);
                }
            } else {
                // this CTA's share of the keys: the unnormalised row, its reference maximum and its sum, where the first tiles were
#pragma unroll
                for (int c = 0; c < AT_D; c += 16) {
                    float part[16];
                    read16(c, part);
#pragma unroll
                    for (int e = 0; e < 16; e += 4)
                        *reinterpret_cast<float4*>(share_o + r * AT_SHARE_LD + c + e) = make_float4(part[e], part[e + 1], part[e + 2], part[e + 3]);
                }
                share_ml[r] = make_float2(m_ref, l_row);
            }
        }
    }
    if (nsplit > 1) {
        // every CTA forms an equal part of the columns from all shares, through the cluster's shared memory
        cg::cluster_group cluster = cg::this_cluster();
        cluster.sync();
        if (warp >= 4) {
            const int r = (tid - 128) & 127;
            const int tok = tok0 + (r >> (__ffs(G) - 1)), head = kvh * G + (r & (G - 1));
            auto merge = [&](auto shares) {
                // eight reads of four columns a thread, whatever the number of shares, all in flight together
                constexpr int NS = decltype(shares)::value, PER = AT_D / 2 / NS;
                const int c0 = split * 2 * PER + ((tid - 128) >> 7) * PER;
                float2 ml[NS];
                float4 o[NS][PER / 4];
#pragma unroll
                for (int sp = 0; sp < NS; ++sp) {
                    ml[sp] = cluster.map_shared_rank(share_ml, sp)[r];
                    const float* from = cluster.map_shared_rank(share_o, sp) + r * AT_SHARE_LD + c0;
#pragma unroll
                    for (int k = 0; k < PER / 4; ++k) o[sp][k] = *reinterpret_cast<const float4*>(from + 4 * k);
                }
                float M = -INFINITY, L = 0.f;
#pragma unroll
                for (int sp = 0; sp < NS; ++sp) M = fmaxf(M, ml[sp].x);
#pragma unroll
                for (int sp = 0; sp < NS; ++sp) {
                    // a row that sees nothing of a share leaves it out (-1); any other takes part, also under a factor of 0: a key or
                    // value that is not finite reaches the rows that see it, whichever CTA walked it
                    ml[sp].x = ml[sp].x == -INFINITY && ml[sp].y == 0.f ? -1.f : fast_exp2(ml[sp].x - M);
                    L = ml[sp].x < 0.f ? L : fmaf(ml[sp].y, ml[sp].x, L);
                }
                const float inv = L > 0.f ? 1.0f / L : 0.f;
                if (r >= rows) return;
#pragma unroll
                for (int k = 0; k < PER / 4; ++k) {
                    const int c = c0 + 4 * k;
                    float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                    for (int sp = 0; sp < NS; ++sp)
#pragma unroll
                        for (int e = 0; e < 4; ++e) v[e] = ml[sp].x < 0.f ? v[e] : fmaf((&o[sp][k].x)[e], ml[sp].x, v[e]);
                    uint2 packed;
                    if (X && opt.gate_mode == 2) {
                        const uint2 raw = *reinterpret_cast<const uint2*>(gate + (size_t)tok * ldg + (size_t)head * AT_D + c);
                        const float2 g0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
                        const float2 g1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
                        packed.x = pack_bf16_pair(v[0] * inv / (1.0f + __expf(-g0.x)), v[1] * inv / (1.0f + __expf(-g0.y)));
                        packed.y = pack_bf16_pair(v[2] * inv / (1.0f + __expf(-g1.x)), v[3] * inv / (1.0f + __expf(-g1.y)));
                    } else {
                        packed.x = pack_bf16_pair(v[0] * inv, v[1] * inv);
                        packed.y = pack_bf16_pair(v[2] * inv, v[3] * inv);
                        if (gate != nullptr) {
                            const float gs = round_as<__nv_bfloat16>(1.0f / (1.0f + expf(-__bfloat162float(gate[(size_t)tok * ldg + head]))));
                            const float2 a = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&packed.x));
                            const float2 b = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&packed.y));
                            packed = make_uint2(pack_bf16_pair(a.x * gs, a.y * gs), pack_bf16_pair(b.x * gs, b.y * gs));
                        }
                    }
                    *reinterpret_cast<uint2*>(out + ((size_t)tok * H + head) * AT_D + c) = packed;
                }
            };
            if (nsplit == 2) merge(std::integral_constant<int, 2>());
            else if (nsplit == 4) merge(std::integral_constant<int, 4>());
            else merge(std::integral_constant<int, 8>());
        }
        cluster.sync();                                  // nobody leaves while its share is read
    }
    // ---- teardown: the tensor memory goes back whatever happened above ----
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 3) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256u) : "memory");
    }
}

}  // namespace

// Whether the tcgen05 prefill kernel takes this shape: head size 64, a group that divides 128.
TK_API int tk_attn_prefill_tc_supported(int H, int Hkv, int D) {
    if (Hkv <= 0 || H % Hkv || D != AT_D) return 0;
    const int G = H / Hkv;
    return G >= 1 && G <= AT_ROWS && AT_ROWS % G == 0;
}

// Tokens of one sequence that a tile of this kernel holds (what the caller cuts portions into).
TK_API int tk_attn_prefill_tc_tokens(int H, int Hkv) { return AT_ROWS / (H / Hkv); }

// 0, or where a CTA gave up waiting on a barrier since the last call (1 and 10 staging, 2-4 MMA issuer,
// 6 and 8 softmax, 9 shared memory out of place). Resets the word.
TK_API int tk_attn_prefill_tc_status() {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_at_error, sizeof(int)) != cudaSuccess) return -1;
    if (v != 0) cudaMemcpyToSymbol(g_at_error, &zero, sizeof(int));
    return v;
}

// q: [T, H, 64] bfloat16; kv_pool: [pages, 2, Hkv, P, 64]; out: [T, H, 64]; tiles of at most
// tk_attn_prefill_tc_tokens tokens of one sequence with consecutive positions; window: see first_seen.
// gate: [T, >= H] bfloat16 with rows ldg apart, the per-head output gate applied to what is
// written (null: none). nsplit > 1: up to that many CTAs (in powers of two, at most 8) share a tile's keys (alternate key tiles;
// each tile takes as many as leave a CTA 8 key tiles), for steps with few tiles and long contexts, where one CTA per tile would
// walk its keys alone on an idle GPU.
// keep_first, sink, gate_mode: see AtOptions (all zero, or gate_mode 1 with a gate: the plain kernel).
TK_API int tk_attn_prefill_tc_opt(const void* q, const void* kv_pool, void* out, const int* positions,
                                  const int* tok_seq, const int* block_table, int bt_stride,
                                  const int* tile_tok0, const int* tile_ntok, int n_tiles, int H, int Hkv, int D,
                                  int P, int window, float scale, const void* gate, int64_t ldg, int nsplit, int keep_first, int sink, int gate_mode,
                                  cudaStream_t stream) {
    TK_CHECK_ARG(keep_first >= 0 && (keep_first == 0 || window > 0), "attn_prefill_tc: kept first positions need a window");
    TK_CHECK_ARG(gate_mode >= 0 && gate_mode <= 2 && (gate_mode == 0) == (gate == nullptr),
                 "attn_prefill_tc: gate mode %d and the gate do not go together", gate_mode);
    TK_CHECK_ARG(gate_mode != 2 || (ldg % 8 == 0 && (uintptr_t)gate % 16 == 0),
                 "attn_prefill_tc: a gate per element is read 16 bytes at a time: rows a multiple of 8 elements "
                 "apart, 16-byte aligned");
    const AtOptions opt{keep_first, sink ? 1 : 0, gate_mode};
    const bool x = keep_first > 0 || sink || gate_mode == 2;
    TK_CHECK_ARG(tk_attn_prefill_tc_supported(H, Hkv, D), "attn_prefill_tc: shape H=%d Hkv=%d D=%d is not taken "
                 "(head size 64, a group that divides 128)", H, Hkv, D);
    TK_CHECK_ARG(P > 0 && n_tiles >= 0, "attn_prefill_tc: bad page size or tile count");
    TK_CHECK_ARG(nsplit >= 1 && (int64_t)n_tiles * Hkv * 8 < 0x7fffffff, "attn_prefill_tc: %d splits of %d tiles", nsplit, n_tiles);
    if (n_tiles == 0) return 0;
    const int split = nsplit >= 8 ? 8 : nsplit >= 4 ? 4 : nsplit >= 2 ? 2 : 1;
    int shift = -1;
    if ((P & (P - 1)) == 0) {
        shift = 0;
        while ((1 << shift) < P) ++shift;
    }
    constexpr size_t smem = AT_SMEM;
    // the pool as rows of 64, boxes of a page or of 64 rows of one; its extent is not known here, and no row is asked for but those of
    // pages that block_table names
    CUtensorMap map = {};
    if (shift >= 3)
        TK_CHECK_ARG(make_map(&map, kv_pool, 0x7fffffff, D, D, shift < 6 ? P : 64), "attn_prefill_tc: cuTensorMapEncodeTiled failed");
    cudaError_t e = cudaFuncSetAttribute(x ? attn_prefill_tc_kernel<true> : attn_prefill_tc_kernel<false>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(n_tiles * Hkv * split);
    cfg.blockDim = dim3(AT_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (tk_pdl_enabled()) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (split > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = split;
        attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
        ++n;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    if (e == cudaSuccess)
        e = cudaLaunchKernelEx(&cfg, x ? attn_prefill_tc_kernel<true> : attn_prefill_tc_kernel<false>, (const __nv_bfloat16*)q,
                               (const __nv_bfloat16*)kv_pool, (__nv_bfloat16*)out, positions, tok_seq, block_table, bt_stride, tile_tok0,
                               tile_ntok, H, Hkv, P, window, scale, shift, map, (const __nv_bfloat16*)gate, ldg, split, opt);
    if (e != cudaSuccess) {
        tk_set_error("attn_prefill_tc: launch failed: %s", cudaGetErrorString(e));
        cudaGetLastError();
        return -2;
    }
    return 0;
}
