// Few-row matrix product of the true 32-bit path: out[M, N] = x[M, K] . W[N, K]^T (+ bias), M <= 8, all
// operands float32, 32-bit FMA sums on the CUDA cores.
//
// Such a product is bound by the stream of weight bytes (eight multiply-adds a weight at most, 128 lanes an SM:
// a third of what the cores can do at the copy bandwidth), so the split is the one that reads every weight row in
// whole 128-byte lines with many loads in flight: a CTA owns 4 weight rows and all of K, its 8 warps take alternate
// 128-wide slices of K, a lane 4 neighbouring columns of all 4 rows, two slices asked for together. The activations
// (64 KB at most for 8 rows of 2,048) are read the same way through L1. A lane then holds 4 x M partial sums; the
// warp adds them up with a halving exchange (31 shuffles for 32 sums instead of 160), the warps through shared memory.
// SWIGLU: the rows of W are all gate rows, then all up rows; the CTA takes 2 channels of both and writes
// silu(gate) * up, so a decoded token needs no activation kernel.
//
// The kernel this replaces up to 8 rows (a 64 x 64 tile of gemm_simt.cu) filled its tile with rows that do not exist
// and ran N / 64 CTAs: the feed-forward of 1,024 x 4,608 at one row took 416 us in three launches, with this kernel
// 15.8 us in two (3.6 TB/s of weights).
#include "common.cuh"

namespace {

constexpr int S32_WARPS = 8, S32_ROWS = 4, S32_SLICE = 128, S32_UNROLL = 2;

__device__ __forceinline__ float4 ld_weights(const float* p) {
    float4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0,%1,%2,%3}, [%4];\n"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "l"(p));
    return v;
}

// Sums v[0 .. V) over the warp, V a power of two up to 32: lane l returns the total of v[l % V].
template <int V>
__device__ __forceinline__ float halving_sum(float (&v)[V], int lane) {
#pragma unroll
    for (int half = V / 2; half >= 1; half /= 2) {
        const bool upper = lane & half;
#pragma unroll
        for (int i = 0; i < half; ++i) {
            const float mine = upper ? v[i + half] : v[i], theirs = upper ? v[i] : v[i + half];
            v[i] = mine + __shfl_xor_sync(0xffffffffu, theirs, half);
        }
    }
    float s = v[0];
#pragma unroll
    for (int o = V; o < 32; o *= 2) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

template <int MT, bool SWIGLU>
__global__ void __launch_bounds__(S32_WARPS * 32)
gemm_stream32_kernel(const float* x, int64_t ldx, const float* __restrict__ w, int64_t ldw,
                     const float* __restrict__ bias, float* out, int64_t ldo, int M, int N, int K) {
    constexpr int V = S32_ROWS * MT;
    __shared__ float red[S32_WARPS][V];
    pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // the CTA's rows of W: 4 neighbours, or 2 gate rows and the up rows of the same channels
    const int channels = SWIGLU ? N / 2 : N;
    constexpr int OWN = SWIGLU ? S32_ROWS / 2 : S32_ROWS;
    const int c0 = blockIdx.x * OWN;
    const float* wr[S32_ROWS];
    int row[S32_ROWS];
#pragma unroll
    for (int r = 0; r < S32_ROWS; ++r) {
        const int c = c0 + r % OWN;
        row[r] = min(c, channels - 1) + (r / OWN) * channels;       // (a row past the end repeats the last one)
        wr[r] = w + (size_t)row[r] * ldw;
    }
    float acc[V];
#pragma unroll
    for (int i = 0; i < V; ++i) acc[i] = 0.f;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    bool waited = false;
    for (int k0 = warp * S32_SLICE; k0 < K; k0 += S32_WARPS * S32_SLICE * S32_UNROLL) {
        float4 wv[S32_UNROLL][S32_ROWS];
#pragma unroll
        for (int u = 0; u < S32_UNROLL; ++u) {
            const int k = k0 + u * S32_WARPS * S32_SLICE + lane * 4;
#pragma unroll
            for (int r = 0; r < S32_ROWS; ++r) wv[u][r] = k < K ? ld_weights(wr[r] + k) : zero;
        }
        if (!waited) {                    // the weights are no kernel's output, the activations are
            pdl_wait();
            waited = true;
        }
#pragma unroll
        for (int u = 0; u < S32_UNROLL; ++u) {
            const int k = k0 + u * S32_WARPS * S32_SLICE + lane * 4;
            if (k >= K) continue;         // (zero weights would turn an infinite activation into NaN)
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                if (m >= M) break;
                const float4 xv = *reinterpret_cast<const float4*>(x + (size_t)m * ldx + k);
#pragma unroll
                for (int r = 0; r < S32_ROWS; ++r) {
                    float a = acc[r * MT + m];
                    a = fmaf(wv[u][r].x, xv.x, a);
                    a = fmaf(wv[u][r].y, xv.y, a);
                    a = fmaf(wv[u][r].z, xv.z, a);
                    acc[r * MT + m] = fmaf(wv[u][r].w, xv.w, a);
                }
            }
        }
    }
    if (!waited) pdl_wait();
    const float total = halving_sum<V>(acc, lane);
    if (lane < V) red[warp][lane] = total;
    __syncthreads();
    const int r = threadIdx.x / MT, m = threadIdx.x % MT;
    if (r < OWN && m < M && c0 + r < channels) {
        float sum = 0.f, up = 0.f;
#pragma unroll
        for (int wv = 0; wv < S32_WARPS; ++wv) {
            sum += red[wv][r * MT + m];
            if (SWIGLU) up += red[wv][(r + OWN) % S32_ROWS * MT + m];
        }
        if (bias != nullptr) {
            sum += bias[c0 + r];
            if (SWIGLU) up += bias[channels + c0 + r];
        }
        out[(size_t)m * ldo + c0 + r] = SWIGLU ? silu_as<float>(sum) * up : sum;
    }
}

template <bool SWIGLU>
void launch_stream32(const float* x, int64_t ldx, const float* w, int64_t ldw, const float* bias, float* out, int64_t ldo,
                     int M, int N, int K, cudaStream_t stream) {
    constexpr int OWN = SWIGLU ? S32_ROWS / 2 : S32_ROWS;
    const dim3 grid(ceil_div(SWIGLU ? N / 2 : N, OWN)), block(S32_WARPS * 32);
#define TK_S32(MT) \
    tk_launch(gemm_stream32_kernel<MT, SWIGLU>, grid, block, 0, stream, x, ldx, w, ldw, bias, out, ldo, M, N, K)
    if (M == 1) TK_S32(1);
    else if (M == 2) TK_S32(2);
    else if (M <= 4) TK_S32(4);
    else TK_S32(8);
#undef TK_S32
}

}  // namespace

TK_API int tk_gemm_stream32_max_rows() { return 8; }

// x: float32 [M, K] rows ldx apart, w: float32 [N, K] rows ldw apart (16-byte aligned rows, K a multiple of 4);
// out: [M, N], or [M, N / 2] with swiglu.
TK_API int tk_gemm_stream32(const void* x, int64_t ldx, const void* w, int64_t ldw, const float* bias, void* out, int64_t ldo,
                            int M, int N, int K, int swiglu, cudaStream_t stream) {
    TK_CHECK_ARG(M > 0 && M <= tk_gemm_stream32_max_rows() && N > 0 && K > 0, "gemm_stream32: M=%d (1..%d) N=%d K=%d", M,
                 tk_gemm_stream32_max_rows(), N, K);
    TK_CHECK_ARG(K % 4 == 0 && ldx % 4 == 0 && ldw % 4 == 0 && (uintptr_t)x % 16 == 0 && (uintptr_t)w % 16 == 0,
                 "gemm_stream32: K and the leading dimensions must be multiples of 4, bases 16-byte aligned");
    TK_CHECK_ARG((M == 1 || ldx >= K) && ldw >= K && (!swiglu || N % 2 == 0) && ldo >= (swiglu ? N / 2 : N),
                 "gemm_stream32: leading dimensions too small, or %d rows of gate and up", N);
    if (swiglu) launch_stream32<true>((const float*)x, ldx, (const float*)w, ldw, bias, (float*)out, ldo, M, N, K, stream);
    else launch_stream32<false>((const float*)x, ldx, (const float*)w, ldw, bias, (float*)out, ldo, M, N, K, stream);
    TK_CHECK_LAUNCH("gemm_stream32");
    return 0;
}
