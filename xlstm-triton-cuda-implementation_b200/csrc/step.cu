// The decoding step: up to STEP_MAX_TOKENS positions of every sequence against a carried state, in one launch.
//
// The carry of mlstm_scan.py:143-195 (operators :15-26) position by position, written out for the few positions of a
// call, with the stabiliser algebra of chunk.cu (A known up front, every weight <= 1):
//     num_t  = exp(A_0 - A_t) scale (q_t S) + sum_{j <= t} exp(a_j - A_t) scale (q_t . k_j) v_j      (b_t: the same with z, 1)
//     S_end  = exp(A_0 - A_T) S + sum_j exp(a_j - A_T) k_j v_j^T                                    (z_end: the same, v dropped)
// and everything is fp32 (gates in double): no operand is rounded to 16 bits on the way.
//
// What bounds it: the state, read once and written once (B = 16, NH = 8, D = 128: 17 MB).  A CTA owns 32 columns (128
// bytes of every row) of one slice's state, so that even a few sequences fill the chip, and holds its piece in registers:
// all of its loads are in flight while the gates and the dot products q . k, q . z are taken, which every CTA of a slice
// does for itself (T (T + 3) / 2 dots of length D).  A row of the state costs 2 T multiply-adds per element, with their
// operands from shared memory: with many sequences a call leaves the memory's time from a few positions on (see below).
// Why up to 16 positions: as far as that it is faster than a block of chunk.cu at every number of sequences.  Kernel time, us,
// bf16, state in and out, at T = 1 | 4 | 5 | 8 | 16 positions, and of the block's launches (which hardly depend on T):
//   D = 128   BH 8: 6 | 8 | 10 | 10 | 19, block 25-27    BH 64: 6 | 8 | 10 | 12 | 21, 35-37    BH 512: 21 | 31 | 58 | 71 | 131, 165-170
//   D = 256   BH 8: 6 | 8 | 10 | 12 | 21, block 33-35    BH 64: 10 | 16 | 21 | 25 | 45, 70      BH 256: 45 | 62 | 80 | 96 | 170, 250
// A call takes at least 40 us, the host's part, against 77 us with the block's five launches.
#include "mlstm_common.cuh"

namespace mlstm {
namespace {

constexpr int STEP_MAX_TOKENS = 16;
constexpr int STEP_THREADS = 256;
constexpr int STEP_COLS = 32;                       // columns of the state per CTA
constexpr int STEP_ROWG = STEP_THREADS / (STEP_COLS / 4);   // threads over the rows (8 lanes of float4 per row)

struct StepArgs {
    const void *q, *k, *v, *f, *i, *o;
    const float *S_in, *z_in;
    const double *F_in, *A_in;
    void* h;
    float *S_out, *z_out;
    double *F_out, *A_out;
    int T;
    float scale;
};

template <typename T16, typename OutT, int D, int TMAX>
__global__ void __launch_bounds__(STEP_THREADS) step_kernel(const StepArgs p) {
    constexpr int NR = D / STEP_ROWG;               // state rows per thread
    constexpr int NW = STEP_THREADS / 32;
    __shared__ __align__(16) T16 sq[TMAX][D], sk[TMAX][D];
    __shared__ __align__(16) float sv[TMAX][STEP_COLS];
    __shared__ float sz[D];
    __shared__ __align__(16) float red[NW][TMAX][STEP_COLS];
    __shared__ float dot[TMAX][TMAX + 1];           // q_t . k_j, and q_t . z in the last column
    __shared__ float w_in[TMAX], w_end[TMAX], wt[TMAX][TMAX], inv_n[TMAX], s_m[TMAX];
    __shared__ double s_a[TMAX], s_A[TMAX];
    __shared__ float s_dec;
    grid_dep_wait();
    grid_dep_launch();
    const int T = p.T, bh = blockIdx.y, col0 = blockIdx.x * STEP_COLS;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int cg = (tid & 7) * 4, rg = tid >> 3;

    const size_t sbase = static_cast<size_t>(bh) * D * D + static_cast<size_t>(rg) * D + col0 + cg;
    float4 s[NR];
#pragma unroll
    for (int j = 0; j < NR; j++)
        s[j] = p.S_in ? *reinterpret_cast<const float4*>(p.S_in + sbase + static_cast<size_t>(j) * STEP_ROWG * D)
                      : make_float4(0.f, 0.f, 0.f, 0.f);
    {
        const size_t xbase = static_cast<size_t>(bh) * T * D;
        const uint4* gq = reinterpret_cast<const uint4*>(static_cast<const T16*>(p.q) + xbase);
        const uint4* gk = reinterpret_cast<const uint4*>(static_cast<const T16*>(p.k) + xbase);
        for (int e = tid; e < T * D / 8; e += STEP_THREADS) {
            reinterpret_cast<uint4*>(&sq[0][0])[e] = gq[e];
            reinterpret_cast<uint4*>(&sk[0][0])[e] = gk[e];
        }
        for (int e = tid; e < T * STEP_COLS; e += STEP_THREADS)
            sv[e / STEP_COLS][e % STEP_COLS] =
                to_f32<T16>(static_cast<const T16*>(p.v)[xbase + static_cast<size_t>(e / STEP_COLS) * D + col0 + e % STEP_COLS]);
        for (int e = tid; e < D; e += STEP_THREADS) sz[e] = p.z_in ? p.z_in[static_cast<size_t>(bh) * D + e] : 0.0f;
    }
    if (warp == 0) {   // the gates (gates.cu has the algebra); lane t: position t
        const double F0 = p.F_in ? p.F_in[bh] : 0.0, A0 = p.A_in ? p.A_in[bh] : -INFINITY;
        double F = 0.0, ig = 0.0;
        if (lane < T) {
            const float x = to_f32<T16>(static_cast<const T16*>(p.f)[static_cast<size_t>(bh) * T + lane]);
            F = static_cast<double>(x < 0.0f ? x - log1pf(expf(x)) : -log1pf(expf(-x)));
            ig = static_cast<double>(to_f32<T16>(static_cast<const T16*>(p.i)[static_cast<size_t>(bh) * T + lane]));
        }
#pragma unroll
        for (int o = 1; o < TMAX; o <<= 1) {
            const double y = __shfl_up_sync(0xffffffffu, F, o);
            if (lane >= o) F += y;
        }
        F += F0;
        const double a = lane < T ? ig - F : -INFINITY;
        double A = fmax(a, A0);
#pragma unroll
        for (int o = 1; o < TMAX; o <<= 1) {
            const double y = __shfl_up_sync(0xffffffffu, A, o);
            if (lane >= o) A = fmax(A, y);
        }
        const double A_end = __shfl_sync(0xffffffffu, A, T - 1);
        // (weights of exactly 0 where there is nothing: no carried state, or an input gate of -inf, however A stands)
        if (lane < T) {
            s_a[lane] = a;
            s_A[lane] = A;
            s_m[lane] = static_cast<float>(F + A);
            w_in[lane] = A0 == -INFINITY ? 0.0f : expf(static_cast<float>(A0 - A));
            w_end[lane] = a == -INFINITY ? 0.0f : expf(static_cast<float>(a - A_end));
        }
        if (lane == T - 1) {
            s_dec = A0 == -INFINITY ? 0.0f : expf(static_cast<float>(A0 - A_end));
            if (blockIdx.x == 0) {
                if (p.F_out) p.F_out[bh] = F;
                if (p.A_out) p.A_out[bh] = A;
            }
        }
    }
    __syncthreads();
    // q_t . k_j (j <= t) and q_t . z, one warp per dot
    for (int e = warp; e < T * (T + 1); e += NW) {
        const int t = e / (T + 1), j = e - t * (T + 1);
        if (j > t && j < T) continue;
        float x = 0.0f;
#pragma unroll
        for (int c = lane; c < D; c += 32) x = fmaf(to_f32<T16>(sq[t][c]), j == T ? sz[c] : to_f32<T16>(sk[j][c]), x);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if (lane == 0) dot[t][j == T ? TMAX : j] = x;
    }
    __syncthreads();
    if (tid < T) {     // the row of weights of position t, its sum and the normaliser
        const int t = tid;
        // (a weight of exactly 0, nothing carried in, also wipes a carried state that is not finite)
        const float w0 = w_in[t] * p.scale;
        float b = w0 == 0.0f ? 0.0f : w0 * dot[t][TMAX];
        for (int j = 0; j <= t; j++) {
            const float w = s_a[j] == -INFINITY ? 0.0f : expf(static_cast<float>(s_a[j] - s_A[t])) * p.scale * dot[t][j];
            wt[t][j] = w;
            b += w;
        }
        w_in[t] = w0;
        inv_n[t] = 1.0f / (fmaxf(fabsf(b), expf(-s_m[t])) + 1e-6f);
    }
    // the state: every position's product with it, and its update
    const float dec = s_dec;
    float4 acc[TMAX];
#pragma unroll
    for (int t = 0; t < TMAX; t++) acc[t] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int j = 0; j < NR; j++) {
        const int row = j * STEP_ROWG + rg;
        float4 n = dec == 0.0f ? make_float4(0.f, 0.f, 0.f, 0.f) : make_float4(dec * s[j].x, dec * s[j].y, dec * s[j].z, dec * s[j].w);
#pragma unroll
        for (int t = 0; t < TMAX; t++) {
            if (t < T) {
                const float qv = to_f32<T16>(sq[t][row]), kv = to_f32<T16>(sk[t][row]) * w_end[t];
                const float4 v4 = *reinterpret_cast<const float4*>(&sv[t][cg]);
                acc[t].x = fmaf(qv, s[j].x, acc[t].x); acc[t].y = fmaf(qv, s[j].y, acc[t].y);
                acc[t].z = fmaf(qv, s[j].z, acc[t].z); acc[t].w = fmaf(qv, s[j].w, acc[t].w);
                n.x = fmaf(kv, v4.x, n.x); n.y = fmaf(kv, v4.y, n.y);
                n.z = fmaf(kv, v4.z, n.z); n.w = fmaf(kv, v4.w, n.w);
            }
        }
        if (p.S_out) *reinterpret_cast<float4*>(p.S_out + sbase + static_cast<size_t>(j) * STEP_ROWG * D) = n;
    }
#pragma unroll
    for (int t = 0; t < TMAX; t++) {
        if (t < T) {
#pragma unroll
            for (int o = 8; o < 32; o <<= 1) {      // the four rows of a warp
                acc[t].x += __shfl_xor_sync(0xffffffffu, acc[t].x, o);
                acc[t].y += __shfl_xor_sync(0xffffffffu, acc[t].y, o);
                acc[t].z += __shfl_xor_sync(0xffffffffu, acc[t].z, o);
                acc[t].w += __shfl_xor_sync(0xffffffffu, acc[t].w, o);
            }
            if (lane < 8) *reinterpret_cast<float4*>(&red[warp][t][cg]) = acc[t];
        }
    }
    if (blockIdx.x == 0 && p.z_out) {
        for (int e = tid; e < D; e += STEP_THREADS) {
            float z = dec == 0.0f ? 0.0f : dec * sz[e];
            for (int t = 0; t < T; t++) z = fmaf(w_end[t], to_f32<T16>(sk[t][e]), z);
            p.z_out[static_cast<size_t>(bh) * D + e] = z;
        }
    }
    __syncthreads();
    for (int e = tid; e < T * STEP_COLS; e += STEP_THREADS) {
        const int t = e / STEP_COLS, c = e % STEP_COLS;
        float x = 0.0f;
#pragma unroll
        for (int w = 0; w < NW; w++) x += red[w][t][c];
        x = w_in[t] == 0.0f ? 0.0f : x * w_in[t];
        for (int j = 0; j <= t; j++) x = fmaf(wt[t][j], sv[j][c], x);
        x *= inv_n[t];
        const size_t at = (static_cast<size_t>(bh) * T + t) * D + col0 + c;
        if (p.o) x *= silu_f(to_f32<T16>(static_cast<const T16*>(p.o)[at]));
        static_cast<OutT*>(p.h)[at] = from_f32<OutT>(x);
    }
}

template <typename T16, typename OutT, int D>
cudaError_t launch_step_d(const StepArgs& a, int BH, cudaStream_t st) {
    const dim3 grid(D / STEP_COLS, BH), block(STEP_THREADS);
    if (a.T == 1) return launch_plain(step_kernel<T16, OutT, D, 1>, grid, block, 0, st, a);
    if (a.T <= 4) return launch_plain(step_kernel<T16, OutT, D, 4>, grid, block, 0, st, a);
    return launch_plain(step_kernel<T16, OutT, D, STEP_MAX_TOKENS>, grid, block, 0, st, a);
}

template <typename T16>
cudaError_t launch_step(const StepArgs& a, int BH, int D, bool h32, cudaStream_t st) {
    if (D == 128) return h32 ? launch_step_d<T16, float, 128>(a, BH, st) : launch_step_d<T16, T16, 128>(a, BH, st);
    return h32 ? launch_step_d<T16, float, 256>(a, BH, st) : launch_step_d<T16, T16, 256>(a, BH, st);
}

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

}  // namespace
}  // namespace mlstm

using namespace mlstm;

extern "C" {

int mlstm_step_max_tokens(void) { return STEP_MAX_TOKENS; }

int mlstm_step(const void* q, const void* k, const void* v, const void* f, const void* i, const void* o, const float* S_in,
               const float* z_in, const double* F_in, const double* A_in, void* h, int h_dtype, float* S_out, float* z_out,
               double* F_out, double* A_out, int B, int NH, int S, int D, int dtype, void* stream) {
    if (!q || !k || !v || !f || !i || !h) return MLSTM_E_ARG;
    if ((S_in == nullptr) != (z_in == nullptr) || (S_in == nullptr) != (F_in == nullptr) || (F_in == nullptr) != (A_in == nullptr))
        return MLSTM_E_ARG;
    if (B <= 0 || NH <= 0 || S <= 0 || D <= 0) return MLSTM_E_ARG;
    if (dtype != MLSTM_DT_F16 && dtype != MLSTM_DT_BF16) return MLSTM_E_UNSUPPORTED;
    if (D != 128 && D != 256) return MLSTM_E_UNSUPPORTED;
    if (S > STEP_MAX_TOKENS || static_cast<long long>(B) * NH > 65535) return MLSTM_E_SHAPE;
    if (h_dtype != MLSTM_DT_F32 && h_dtype != dtype) return MLSTM_E_ARG;
    if (!aligned16(q) || !aligned16(k) || !aligned16(v) || !aligned16(o) || !aligned16(h) || !aligned16(S_in) || !aligned16(z_in) ||
        !aligned16(S_out))
        return MLSTM_E_ALIGN;
    StepArgs a{q, k, v, f, i, o, S_in, z_in, F_in, A_in, h, S_out, z_out, F_out, A_out, S, 1.0f / sqrtf(static_cast<float>(D))};
    const bool h32 = h_dtype == MLSTM_DT_F32;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const cudaError_t ce = dtype == MLSTM_DT_BF16 ? launch_step<__nv_bfloat16>(a, B * NH, D, h32, st) : launch_step<__half>(a, B * NH, D, h32, st);
    if (ce != cudaSuccess) cudaGetLastError();
    return ce == cudaSuccess ? MLSTM_OK : note_cuda_error(ce, "launch of step_kernel");
}

}  // extern "C"
