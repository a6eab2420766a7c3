// out[M, N] = x[M, K] . W[N, K]^T (+ bias), all float32, on the bfloat16 tensor cores with the errors of 32-bit sums:
//
//   every operand is taken apart as x = h + m + l, three bfloat16 numbers of 8 significant bits each (h = bf16(x), m =
//   bf16(x - h), l = bf16(x - h - m): the differences are exact), and of the nine products the six that reach 2^-24 of
//   the whole are formed, h h', h m', m h', m m', h l', l h'. Each is exact in the tensor core; what is left out is below
//   2^-26. (Inputs below 2^-110 in size lose the low bits of l to underflow.)
//
//   A tensor core adds a product to its accumulator with truncation, one step per 16 columns of K, and the losses all pull
//   one way: over K = 2,048 the plain bfloat16 product is off by 2.1e-6 where a chain of 32-bit multiply-adds is off by
//   0.4e-6. So h h', which carries the size of the result, is summed in the tensor core over 128 columns only (about
//   1e-7) and then joins sums that live in registers, rounded to nearest; the five small products have an accumulator of
//   their own, 2^-8 of the size, whose losses are as much smaller, and join once at the end. Off by 1.3e-7 to 2.5e-7
//   against 64 bits (normal values, K 1,024 to 10,752), where the multiply-adds of gemm_simt.cu are off by 0.6e-6 to 1.9e-6.
//
// Bound by the tensor pipe: six bfloat16 products, i.e. a sixth of its rate, against which the CUDA cores' multiply-adds
// have a twentieth: 2,048 x 16,384 x 2,048 in 694 us (198 TFLOP/s; gemm_simt.cu 5,414), 16 x 2,048 x 2,048 in 15.5 us (119),
// never slower than it from 9 rows and 128 x 128 weights on (9 x 256 x 256 9.4 us against 15.8; taken from 256 x 256 on). A CTA owns
// 128 rows of W (the MMA's M) and BN tokens; 16 warps read 32 columns of both operands from memory into registers a chunk
// ahead, take them apart and store the three parts as K-major tiles in the 128-byte swizzle (h and m side by side in one row, l in a tile that the two buffers share by halves), one thread issues the
// twelve MMAs of a chunk, and all warps work on the next chunk meanwhile. BN = 256 keeps shared memory (96 bytes a cycle
// of operand reads) below what the MMAs would need at 128 columns (128). The tokens' tiles are the grid's fast axis, so
// that neighbouring CTAs read the same rows of W from L2. A product with few tiles is split along K over a cluster whose
// CTAs add up their parts through distributed shared memory in a fixed order.
//
// An input that is infinite, NaN or rounds up to infinity in 16 bits leaves NaN in every sum it enters, and finite inputs
// whose products overflow may leave infinities of both signs in the two accumulators: a sum that does not come out finite is
// formed again by multiply-adds in the order of K, which put infinities and NaN where gemm_simt.cu puts them.
#include <cooperative_groups.h>

#include "parts.cuh"
#include "tcgen05.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr int SP_THREADS = 512, SP_WARPS = 16, SP_BM = 128, SP_KC = 32, SP_GROUP = 4;   // SP_GROUP chunks a sum in the tensor core

__device__ int g_split_error = 0;

__device__ __forceinline__ bool split_wait(uint32_t bar, uint32_t parity, int where) {
    const long long start = clock64();
    while (!mbar_try_wait(bar, parity)) {
        if (clock64() - start > 2000000000LL) {
            atomicCAS(&g_split_error, 0, where);
            return false;
        }
    }
    return true;
}

template <int COLS>
__device__ __forceinline__ void tmem_add(uint32_t taddr, float (&acc)[COLS]) {
    if constexpr (COLS >= 32) {
#pragma unroll
        for (int c = 0; c < COLS; c += 32) {
            float v[32];
            tmem_ld32(taddr + c, v);
#pragma unroll
            for (int e = 0; e < 32; ++e) acc[c + e] += v[e];
        }
    } else {
#pragma unroll
        for (int c = 0; c < COLS; c += 8) {
            float v[8];
            tmem_ld8(taddr + c, v);
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[c + e] += v[e];
        }
    }
}

// One element by multiply-adds in the order of K.
__device__ __noinline__ float sum_again(const float* w, int64_t ldw, int row, const float* x, int64_t ldx, int token, int K) {
    const float *wr = w + (size_t)row * ldw, *xr = x + (size_t)token * ldx;
    float s = 0.f;
    for (int k = 0; k < K; ++k) s = fmaf(wr[k], xr[k], s);
    return s;
}

template <int BN>
__global__ void __launch_bounds__(SP_THREADS, BN <= 64 ? 2 : 1)
gemm_split32_kernel(const float* x, int64_t ldx, const float* w, int64_t ldw, const float* __restrict__ bias, float* out,
                    int64_t ldo, int M, int N, int K, int splitk) {
    constexpr int ROWS = SP_BM + BN, UNITS = (ROWS * 4 + SP_THREADS - 1) / SP_THREADS;
    constexpr int TILE = ROWS * 128;                    // bytes of one tile: 64 bfloat16 of every row
    constexpr int COLS = BN / 4;                        // accumulator columns a thread keeps
    constexpr uint32_t TMEM_COLS = 2 * BN;              // h h' | the small products
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bar_store[2];
    __shared__ uint32_t tmem_slot;
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t tile_l = base + 2 * TILE;
    const uint32_t bar0 = smem_u32(&bar_store[0]);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tok0 = blockIdx.x * BN, row0 = blockIdx.y * SP_BM;
    const int chunks_all = (K + SP_KC - 1) / SP_KC, per = (chunks_all + splitk - 1) / splitk;
    const int first = blockIdx.z * per, n_chunks = max(0, min(chunks_all, first + per) - first);

    pdl_launch_dependents();
    if (tid == 0) {
        mbar_init(bar0, 1);
        mbar_init(bar0 + 8, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_main = *(volatile uint32_t*)&tmem_slot, tmem_corr = tmem_main + BN;

    // A unit is 8 neighbouring floats of one row: lane -> (row of a group of 8, 16-byte chunk of its 4), ordered so that
    // the eight lanes of a 16-byte store phase (rows r and r + 4) meet eight different banks
    const int sub_row = ((lane >> 2) >> 1) + ((lane >> 2) & 1) * 4, c8 = lane & 3;
    const float* src[UNITS];
    bool live[UNITS];
#pragma unroll
    for (int i = 0; i < UNITS; ++i) {
        const int r = (warp + SP_WARPS * i) * 8 + sub_row;
        const bool is_w = i == 0;                       // (the first 16 groups of 8 rows are W's)
        const int g = is_w ? row0 + r : tok0 + r - SP_BM;
        live[i] = r < ROWS && g < (is_w ? N : M);
        src[i] = (is_w ? w + (size_t)(live[i] ? g : 0) * ldw : x + (size_t)(live[i] ? g : 0) * ldx) + c8 * 8;
    }
    float4 next[UNITS][2];
    auto fetch = [&](int chunk) {
        const int k = chunk * SP_KC + c8 * 8;
#pragma unroll
        for (int i = 0; i < UNITS; ++i)
#pragma unroll
            for (int e = 0; e < 2; ++e)
                next[i][e] = live[i] && k + 4 * e < K ? *reinterpret_cast<const float4*>(src[i] + chunk * SP_KC + 4 * e)
                                                      : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    float acc[COLS];
#pragma unroll
    for (int c = 0; c < COLS; ++c) acc[c] = 0.f;
    const uint32_t my_tmem = ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)((warp >> 2) * COLS);
    bool ok = true;

    pdl_wait();
    if (n_chunks > 0) fetch(first);
    for (int c = 0; c < n_chunks; ++c) {
        const int b = c & 1;
        const uint32_t tile_hm = base + b * TILE;
        if (c >= 2 && ok) ok = split_wait(bar0 + 8 * b, ((c >> 1) - 1) & 1, 11);     // the MMAs that read this buffer are done
#pragma unroll
        for (int i = 0; i < UNITS; ++i) {
            if ((warp + SP_WARPS * i) * 8 >= ROWS) continue;
            uint4 h, m, l;
            take_apart(next[i][0].x, next[i][0].y, h.x, m.x, l.x);
            take_apart(next[i][0].z, next[i][0].w, h.y, m.y, l.y);
            take_apart(next[i][1].x, next[i][1].y, h.z, m.z, l.z);
            take_apart(next[i][1].z, next[i][1].w, h.w, m.w, l.w);
            const uint32_t row_at = (uint32_t)((warp + SP_WARPS * i) * 8 + sub_row) * 128;
            auto put = [&](uint32_t tile, uint32_t chunk16, const uint4& v) {        // (sub_row is the row modulo 8)
                asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(tile + row_at + ((chunk16 ^ sub_row) << 4)), "r"(v.x),
                             "r"(v.y), "r"(v.z), "r"(v.w)
                             : "memory");
            };
            put(tile_hm, c8, h);
            put(tile_hm, 4 + c8, m);
            put(tile_l, 4 * b + c8, l);
        }
        if (c + 1 < n_chunks) fetch(first + c + 1);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        constexpr uint32_t idesc = umma_idesc(BN);
        const uint64_t hm_w = umma_desc(tile_hm), hm_x = umma_desc(tile_hm + SP_BM * 128);
        if (tid == 0) {
            const uint64_t l_w = umma_desc(tile_l) + 4 * b, l_x = umma_desc(tile_l + SP_BM * 128) + 4 * b;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (int k = 0; k < 2; ++k) {                                      // 16 columns (32 bytes) a step
                umma_bf16(tmem_corr, hm_w + 2 * k, l_x + 2 * k, idesc, (c > 0 || k > 0) ? 1u : 0u);
                umma_bf16(tmem_corr, l_w + 2 * k, hm_x + 2 * k, idesc, 1u);
                umma_bf16(tmem_corr, hm_w + 4 + 2 * k, hm_x + 4 + 2 * k, idesc, 1u);
                umma_bf16(tmem_corr, hm_w + 2 * k, hm_x + 4 + 2 * k, idesc, 1u);
                umma_bf16(tmem_corr, hm_w + 4 + 2 * k, hm_x + 2 * k, idesc, 1u);
            }
        }
        if (c > 0 && c % SP_GROUP == 0) {
            // the sums of the group before move to registers while the small products run
            __syncwarp();
            if (ok) ok = split_wait(bar0 + 8 * (b ^ 1), ((c - 1) >> 1) & 1, 12);
            __syncwarp();
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            tmem_add<COLS>(tmem_main + my_tmem, acc);
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncthreads();
        }
        if (tid == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (int k = 0; k < 2; ++k)
                umma_bf16(tmem_main, hm_w + 2 * k, hm_x + 2 * k, idesc, (c % SP_GROUP > 0 || k > 0) ? 1u : 0u);
            umma_commit(bar0 + 8 * b);
        }
        __syncwarp();
    }
    if (n_chunks > 0) {
        const int c = n_chunks - 1;
        if (ok) ok = split_wait(bar0 + 8 * (c & 1), (c >> 1) & 1, 13);
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        tmem_add<COLS>(tmem_main + my_tmem, acc);
        tmem_add<COLS>(tmem_corr + my_tmem, acc);
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
    __syncthreads();
    const int i_row = row0 + (warp & 3) * 32 + lane, col0 = (warp >> 2) * COLS;
    if (splitk == 1) {
        if (i_row < N) {
            const float add = bias != nullptr ? bias[i_row] : 0.f;
#pragma unroll
            for (int c = 0; c < COLS; ++c)
                if (tok0 + col0 + c < M) {
                    if (!isfinite(acc[c])) acc[c] = sum_again(w, ldw, i_row, x, ldx, tok0 + col0 + c, K);
                    out[(size_t)(tok0 + col0 + c) * ldo + i_row] = acc[c] + add;
                }
        }
    } else {
        // every CTA of the cluster leaves its part [BN][128] in its own shared memory (the operand tiles are done with);
        // each adds up a share of the tokens over all parts
        cg::cluster_group cluster = cg::this_cluster();
        float* mine = reinterpret_cast<float*>(smem_raw + (base - smem_u32(smem_raw)));
        const int r = (warp & 3) * 32 + lane;
#pragma unroll
        for (int c = 0; c < COLS; ++c) mine[(col0 + c) * SP_BM + r] = acc[c];
        cluster.sync();
        const int share = BN / splitk, from = (int)cluster.block_rank() * share;
        const float add = bias != nullptr && i_row < N ? bias[i_row] : 0.f;
        for (int j = from + (warp >> 2); j < from + share; j += 4) {
            float s = 0.f;
            for (int p = 0; p < splitk; ++p) s += cluster.map_shared_rank(mine, p)[j * SP_BM + r];
            if (i_row >= N || tok0 + j >= M) continue;
            if (!isfinite(s)) s = sum_again(w, ldw, i_row, x, ldx, tok0 + j, K);
            out[(size_t)(tok0 + j) * ldo + i_row] = s + add;
        }
        cluster.sync();
    }
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_main), "r"(TMEM_COLS) : "memory");
    }
}

template <int BN>
cudaError_t launch_split32(const float* x, int64_t ldx, const float* w, int64_t ldw, const float* bias, float* out, int64_t ldo,
                           int M, int N, int K, int splitk, cudaStream_t stream) {
    const size_t smem = (size_t)(SP_BM + BN) * 128 * 3 + 1024;
    const cudaError_t raised =
        cudaFuncSetAttribute(gemm_split32_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (raised != cudaSuccess) return raised;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((M + BN - 1) / BN, (N + SP_BM - 1) / SP_BM, splitk);
    cfg.blockDim = dim3(SP_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (tk_pdl_enabled()) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (splitk > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = 1;
        attr[n].val.clusterDim.y = 1;
        attr[n++].val.clusterDim.z = splitk;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, gemm_split32_kernel<BN>, x, ldx, w, ldw, bias, out, ldo, M, N, K, splitk);
}

}  // namespace

// 0 if no such product on the current device has given up on a barrier since the last call. Resets the word.
TK_API int tk_gemm_split32_status() {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_split_error, sizeof(int)) != cudaSuccess) return -1;
    if (v != 0) cudaMemcpyToSymbol(g_split_error, &zero, sizeof(int));
    return v;
}

// x: float32 [M, K] rows ldx apart, w: float32 [N, K] rows ldw apart (16-byte aligned rows, K a multiple of 4), out:
// float32 [M, N] rows ldo apart.
TK_API int tk_gemm_split32(const void* x, int64_t ldx, const void* w, int64_t ldw, const float* bias, void* out, int64_t ldo,
                           int M, int N, int K, cudaStream_t stream) {
    TK_CHECK_ARG(M > 0 && N > 0 && K > 0 && ldx >= K && ldw >= K && ldo >= N, "gemm_split32: bad sizes M=%d N=%d K=%d", M, N, K);
    TK_CHECK_ARG(K % 4 == 0 && ldx % 4 == 0 && ldw % 4 == 0 && (uintptr_t)x % 16 == 0 && (uintptr_t)w % 16 == 0,
                 "gemm_split32: K and the leading dimensions must be multiples of 4, bases 16-byte aligned");
    TK_CHECK_ARG((N + SP_BM - 1) / SP_BM <= 65535, "gemm_split32: N=%d", N);
    const int groups = ceil_div(K, SP_KC * SP_GROUP);
    // more than 128 tokens in tiles of 256, but for a K too short to be split while tiles of 128 all run at once: those tiles
    // are the only way to more of the GPU then (256 to 1,000 x 300 x 300: 22.9 us in tiles of 256, gemm_simt.cu 21.3, 15.0 in
    // tiles of 128; from 129 x 256 x 384 to 2,048 x 1,000 x 256 26.3 to 63.1 there, 15.6 and 13.0 here)
    const bool small = groups < 4 && ceil_div(M, 128) * ceil_div(N, SP_BM) <= 148;
    const int BN = M <= 32 ? 32 : M <= 64 ? 64 : M <= 128 || small ? 128 : 256;
    const int tiles = ceil_div(M, BN) * ceil_div(N, SP_BM);
    // K is split while the CTAs fill no more than the GPU (two of them an SM up to 64 tokens) and each keeps 256 columns
    const int room = BN <= 64 ? 2 * 148 : 148;
    int splitk = 1;
    while (splitk < 8 && tiles * splitk * 2 <= room && groups / (splitk * 2) >= 2) splitk *= 2;
    cudaError_t e;
#define TK_SPLIT(BN_) \
    e = launch_split32<BN_>((const float*)x, ldx, (const float*)w, ldw, bias, (float*)out, ldo, M, N, K, splitk, stream)
    if (BN == 32) TK_SPLIT(32);
    else if (BN == 64) TK_SPLIT(64);
    else if (BN == 128) TK_SPLIT(128);
    else TK_SPLIT(256);
#undef TK_SPLIT
    if (e != cudaSuccess) {
        tk_set_error("gemm_split32: launch failed: %s", cudaGetErrorString(e));
        cudaGetLastError();
        return -2;
    }
    return 0;
}
