// The parallel mLSTM in fp32 on the CUDA cores in two stages (fp32 inputs at head dimensions the tensor-core forms do not
// take; the contractions of mlstm_matmul.py:37-101 and 200-316 in the arithmetic of its tl.dot(..., allow_tf32=False)):
//     GATE    W = (X Y^T + g) * exp2(ec + er) for the causal 64 x 64 tiles, fp32, to scratch
//     APPLY   out = W Z, or W^T Z (TRANS), over the causal side, with the pass' epilogue
// mm_simt.cu forms the gated tile again for every 64 output columns and every pass (at D = 256 forward and backward execute
// 20 contractions); here each is executed once (2 and 5, the algorithmic count; the backward's two matrices serve three
// results).  The sums are the same fp32 FMA sums.
// One gated matrix for two results fixes which side's exponent is rounded first, which had moved dK, dV and dI 4 to 34 % away from
// 64 bits against the one-stage passes at f ~ N(1, 1).  Row and column parts therefore carry the rests of their rounding (gAn_lo
// of the gate pass): errors are 0.15 - 0.6 of the one-stage ones at f ~ N(1, 1), 0.15 - 0.93 at N(0, 1), 0.74 - 0.98 at N(3, 1)
// (2-norm of h, dQ, dK, dV, dI; S 128 - 1664, D 32, 96, 256).  It costs 1 % (B = 1, NH = 4, S = 1024, D = 256: 104.3 -> 104.5 | 225.7 -> 228.7 us).
//
// What bounds it: the FMA units.  64 x 64 tiles on 128 threads of 8 x 4 results: per k step 32 FMA (8 cycles of an SM's
// four schedulers for the CTA's four warps) against about 4 cycles of shared-memory reads; small tiles because a few heads
// at S = 1024 are all the parallelism there is (B = 1, NH = 4: 544 GATE tiles, 256 APPLY tiles).
// Measured, fp32, us, one stage -> two, forward | backward: B = 1, NH = 4, S = 1024, D = 256 388 -> 109 | 1165 -> 234;
// B = 2, NH = 8, S = 2048, D = 256 3364 -> 931 | 10062 -> 2209 (37 and 39 TFLOP/s); B = 1, NH = 8, S = 2048, D = 32
// 250 -> 184 | 736 -> 401; B = 1, NH = 1, S = 128, D = 32 32 -> 34 | 60 -> 43 (launches).
#include "mlstm_common.cuh"

namespace mlstm {
namespace {

constexpr int GT = 64;          // tile edge; one reference block of the gate vectors
constexpr int GK = 16;          // contraction chunk
constexpr int GTHREADS = 128;
constexpr int LDS_T = GT + 4;   // shared-memory row (float4-aligned, staggered banks)
static_assert(GT == REF_BLOCK, "one column reference per tile");

template <typename T>
__device__ __forceinline__ float4 load4(const T* p) {
    if constexpr (sizeof(T) == 4) {
        return *reinterpret_cast<const float4*>(p);
    } else {
        const uint2 raw = *reinterpret_cast<const uint2*>(p);
        const T* e = reinterpret_cast<const T*>(&raw);
        return make_float4(to_f32<T>(e[0]), to_f32<T>(e[1]), to_f32<T>(e[2]), to_f32<T>(e[3]));
    }
}

// One operand's chunk in shared memory, [GK][LDS_T] (contraction index first).  KMAJOR: the source's rows are the operand's
// rows and run along the contraction; else the source's rows are the contraction.  Out of range reads as zero.
template <typename T, bool KMAJOR>
struct Operand {
    const T* base;      // first row of the tile (KMAJOR) or first contraction row, first column
    size_t ld;
    int rows, cols;     // what may be read, from base: KMAJOR rows x contraction; else contraction rows x columns
    float4 r[2];
    __device__ __forceinline__ void fetch(int k0) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int e = threadIdx.x + h * GTHREADS;
            const int row = KMAJOR ? (e >> 2) : k0 + (e >> 4), col = KMAJOR ? k0 + (e & 3) * 4 : (e & 15) * 4;
            r[h] = (row < rows && col < cols) ? load4<T>(base + static_cast<size_t>(row) * ld + col) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
    __device__ __forceinline__ void put(float (*s)[LDS_T]) const {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int e = threadIdx.x + h * GTHREADS;
            if constexpr (KMAJOR) {
                const int row = e >> 2, k = (e & 3) * 4;
                s[k][row] = r[h].x; s[k + 1][row] = r[h].y; s[k + 2][row] = r[h].z; s[k + 3][row] = r[h].w;
            } else {
                *reinterpret_cast<float4*>(&s[e >> 4][(e & 15) * 4]) = r[h];
            }
        }
    }
};

// acc[8][4] += A B over k in [0, kn): this thread's rows 8 ty .. and columns 4 tx ..
template <typename OpA, typename OpB>
__device__ __forceinline__ void contract(OpA& a, OpB& b, int kn, float (*sA)[GK][LDS_T], float (*sB)[GK][LDS_T], float (&acc)[8][4]) {
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    a.fetch(0);
    b.fetch(0);
    a.put(sA[0]);
    b.put(sB[0]);
    __syncthreads();
    int buf = 0;
    for (int k0 = 0; k0 < kn; k0 += GK, buf ^= 1) {
        const bool more = k0 + GK < kn;
        if (more) {
            a.fetch(k0 + GK);
            b.fetch(k0 + GK);
        }
#pragma unroll
        for (int k = 0; k < GK; k++) {
            float x[8], y[4];
            *reinterpret_cast<float4*>(&x[0]) = *reinterpret_cast<const float4*>(&sA[buf][k][ty * 8]);
            *reinterpret_cast<float4*>(&x[4]) = *reinterpret_cast<const float4*>(&sA[buf][k][ty * 8 + 4]);
            *reinterpret_cast<float4*>(&y[0]) = *reinterpret_cast<const float4*>(&sB[buf][k][tx * 4]);
#pragma unroll
            for (int i = 0; i < 8; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = fmaf(x[i], y[j], acc[i][j]);
        }
        if (more) {
            a.put(sA[buf ^ 1]);
            b.put(sB[buf ^ 1]);
        }
        __syncthreads();
    }
}

struct GateProblem {
    const void *X, *Y;          // query-side and key-side operand, [BH, S, D]
    const float* g;             // additive term per row, or nullptr
    float* W;                   // [slices][Sp][Sp]
    float* bpart;               // [slices][NT][Sp] row sums per tile column, or nullptr
};
struct GateArgs {
    GateProblem pr[2];
    const float *row_rel, *col_rel, *row_lo, *col_lo;
    const double *row_ref, *col_ref;
    float er_add;
    int S, Spad, D, Sp, bh0;
};

template <typename T>
__global__ void __launch_bounds__(GTHREADS) simt_gate_kernel(const GateArgs p) {
    __shared__ __align__(16) float sA[2][GK][LDS_T], sB[2][GK][LDS_T];
    grid_dep_wait();
    grid_dep_launch();
    const GateProblem& pr = p.pr[blockIdx.z];
    int rt = static_cast<int>((sqrtf(8.0f * blockIdx.x + 1.0f) - 1.0f) * 0.5f);
    while ((rt + 1) * (rt + 2) / 2 <= static_cast<int>(blockIdx.x)) rt++;      // (the root is rounded)
    while (rt * (rt + 1) / 2 > static_cast<int>(blockIdx.x)) rt--;
    const int ct = blockIdx.x - rt * (rt + 1) / 2;
    const int slice = blockIdx.y, bh = p.bh0 + slice;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    float acc[8][4] = {};
    Operand<T, true> a{static_cast<const T*>(pr.X) + (static_cast<size_t>(bh) * p.S + rt * GT) * p.D, static_cast<size_t>(p.D), p.S - rt * GT, p.D, {}};
    Operand<T, true> b{static_cast<const T*>(pr.Y) + (static_cast<size_t>(bh) * p.S + ct * GT) * p.D, static_cast<size_t>(p.D), p.S - ct * GT, p.D, {}};
    contract(a, b, p.D, sA, sB, acc);

    const size_t vec = static_cast<size_t>(bh) * p.Spad, ref = static_cast<size_t>(bh) * (p.Spad / REF_BLOCK);
    const double refs = p.row_ref[ref + rt] + p.col_ref[ref + ct] + static_cast<double>(p.er_add);
    const int col0 = ct * GT + tx * 4;
    const float4 ec4 = *reinterpret_cast<const float4*>(p.col_rel + vec + col0);
    const float4 el4 = *reinterpret_cast<const float4*>(p.col_lo + vec + col0);
    const float ec[4] = {ec4.x, ec4.y, ec4.z, ec4.w}, el[4] = {el4.x, el4.y, el4.z, el4.w};
    float* W = pr.W + static_cast<size_t>(slice) * p.Sp * p.Sp;
    float row_rel[8], row_lo[8];      // (the loads of all rows in front of the first use)
#pragma unroll
    for (int i = 0; i < 8; i++) {
        row_rel[i] = p.row_rel[vec + rt * GT + ty * 8 + i];
        row_lo[i] = p.row_lo[vec + rt * GT + ty * 8 + i];
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int row = rt * GT + ty * 8 + i;
        // row and column part of the exponent as two floats each: they may be 60 and -60 where their sum is of order 1, and a
        // rounding of the 60 would be a relative error of 2^-19 of the weight
        const double er_d = static_cast<double>(row_rel[i]) + refs;
        const float er = static_cast<float>(er_d);
        const float er_lo = er == -INFINITY ? 0.0f : static_cast<float>(er_d - er) + row_lo[i];
        const float g = pr.g ? pr.g[vec + row] : 0.0f;
        float w[4], sum = 0.0f;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            w[j] = (acc[i][j] + g) * exp2f((ec[j] + er) + (el[j] + er_lo));
            if (col0 + j > row || row >= p.S) w[j] = 0.0f;       // (a valid row's causal columns are valid)
            sum += w[j];
        }
        *reinterpret_cast<float4*>(W + static_cast<size_t>(row) * p.Sp + col0) = make_float4(w[0], w[1], w[2], w[3]);
        if (pr.bpart) {
#pragma unroll
            for (int o = 1; o < 16; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            if (tx == 0) pr.bpart[(static_cast<size_t>(slice) * (p.Sp / GT) + ct) * p.Sp + row] = sum;
        }
    }
}

struct ApplyProblem {
    const float* W;
    const void* Z;              // [BH, S, D]
    void* out;                  // [BH, S, D]
    const void* dot_src;        // rows are dotted with this, or nullptr
    float* dot_out;             // [D / 64 rounded up][BH, Spad] partial dots, dot_stride apart
};
struct ApplyArgs {
    ApplyProblem pr[2];
    const float* bpart;         // forward: normalise by the row sums
    const float* m;
    float* b_out;
    const void* ogate;
    long long dot_stride;
    int S, Spad, D, Sp, bh0;
};

template <typename T, typename OutT, bool TRANS, bool FWD_EPI>
__global__ void __launch_bounds__(GTHREADS) simt_apply_kernel(const ApplyArgs p) {
    __shared__ __align__(16) float sA[2][GK][LDS_T], sB[2][GK][LDS_T];
    __shared__ float s_inv[GT];
    grid_dep_wait();
    grid_dep_launch();
    const int NT = p.Sp / GT, nv = (p.D + GT - 1) / GT;
    const int nprob = gridDim.z;
    // longest contractions first; neighbouring blocks share the rows of W
    const int prob = nprob == 1 ? 0 : blockIdx.z;
    const ApplyProblem& pr = p.pr[prob];
    const int w = blockIdx.x / nv, vt = blockIdx.x - w * nv;
    const int mt = TRANS ? w : NT - 1 - w;
    const int slice = blockIdx.y, bh = p.bh0 + slice;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const float* W = pr.W + static_cast<size_t>(slice) * p.Sp * p.Sp;
    const size_t base = static_cast<size_t>(bh) * p.S * p.D;
    const int k0 = TRANS ? mt * GT : 0, kn = TRANS ? p.Sp - k0 : (mt + 1) * GT;
    if (FWD_EPI && threadIdx.x < GT) {
        const int row = mt * GT + threadIdx.x;
        float b = 0.0f;
        for (int c = 0; c <= mt; c++) b += p.bpart[(static_cast<size_t>(slice) * NT + c) * p.Sp + row];
        const bool ok = row < p.S;
        const size_t at = static_cast<size_t>(bh) * p.S + row;
        s_inv[threadIdx.x] = ok ? 1.0f / (fmaxf(fabsf(b), expf(-p.m[at])) + 1e-6f) : 0.0f;
        if (ok && vt == 0 && p.b_out) p.b_out[at] = b;
    }
    float acc[8][4] = {};
    Operand<T, false> z{static_cast<const T*>(pr.Z) + base + static_cast<size_t>(k0) * p.D + vt * GT, static_cast<size_t>(p.D), p.S - k0, p.D - vt * GT, {}};
    if constexpr (TRANS) {
        Operand<float, false> a{W + static_cast<size_t>(k0) * p.Sp + mt * GT, static_cast<size_t>(p.Sp), kn, GT, {}};
        contract(a, z, kn, sA, sB, acc);
    } else {
        Operand<float, true> a{W + static_cast<size_t>(mt) * GT * p.Sp, static_cast<size_t>(p.Sp), GT, kn, {}};
        contract(a, z, kn, sA, sB, acc);
    }
    const int d = vt * GT + tx * 4;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int row = mt * GT + ty * 8 + i;
        const bool ok = row < p.S && d < p.D;
        const size_t at = base + static_cast<size_t>(row) * p.D + d;
        float x[4] = {acc[i][0], acc[i][1], acc[i][2], acc[i][3]};
        if (FWD_EPI) {
            const float inv = s_inv[ty * 8 + i];
#pragma unroll
            for (int j = 0; j < 4; j++) x[j] *= inv;
        }
        float dot = 0.0f;
        if (ok) {
            if (FWD_EPI && p.ogate) {
                const float4 o = load4<T>(static_cast<const T*>(p.ogate) + at);
                x[0] *= silu_f(o.x); x[1] *= silu_f(o.y); x[2] *= silu_f(o.z); x[3] *= silu_f(o.w);
            }
            if (!FWD_EPI && pr.dot_src) {
                const float4 s = load4<T>(static_cast<const T*>(pr.dot_src) + at);
                dot = (x[0] * s.x + x[1] * s.y) + (x[2] * s.z + x[3] * s.w);
            }
            OutT* out = static_cast<OutT*>(pr.out) + at;
            if constexpr (sizeof(OutT) == 4) {
                *reinterpret_cast<float4*>(out) = make_float4(x[0], x[1], x[2], x[3]);
            } else {
                __align__(8) OutT v[4] = {from_f32<OutT>(x[0]), from_f32<OutT>(x[1]), from_f32<OutT>(x[2]), from_f32<OutT>(x[3])};
                *reinterpret_cast<uint2*>(out) = *reinterpret_cast<const uint2*>(v);
            }
        }
        if (!FWD_EPI && pr.dot_out) {
#pragma unroll
            for (int o = 1; o < 16; o <<= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
            if (tx == 0 && row < p.S) pr.dot_out[vt * p.dot_stride + static_cast<long long>(bh) * p.Spad + row] = dot;
        }
    }
}

inline int sp_of(int S) { return round_up(S, GT); }

template <typename T, typename OutT>
int fwd_launch(const SimtGemmArgs& a, const void* q, const void* k, const void* v, const void* o, void* h, cudaStream_t st) {
    const int Sp = sp_of(a.S), NT = Sp / GT, group = simt_gemm_group(a.BH, a.S);
    for (int bh0 = 0; bh0 < a.BH; bh0 += group) {
        const int n = a.BH - bh0 < group ? a.BH - bh0 : group;
        GateArgs g{};
        g.pr[0] = GateProblem{q, k, nullptr, a.W0, a.W0 + static_cast<size_t>(group) * Sp * Sp};
        g.row_rel = a.gAn; g.row_ref = a.An_ref; g.col_rel = a.ga; g.col_ref = a.a_ref; g.row_lo = a.gAn_lo; g.col_lo = a.ga_lo;
        g.er_add = -0.5f * log2f(static_cast<float>(a.D));
        g.S = a.S; g.Spad = a.Spad; g.D = a.D; g.Sp = Sp; g.bh0 = bh0;
        if (launch_plain(simt_gate_kernel<T>, dim3(NT * (NT + 1) / 2, n, 1), dim3(GTHREADS), 0, st, g) != cudaSuccess) return MLSTM_E_CUDA;
        ApplyArgs p{};
        p.pr[0] = ApplyProblem{a.W0, v, h, nullptr, nullptr};
        p.bpart = g.pr[0].bpart; p.m = a.m; p.b_out = a.b; p.ogate = o;
        p.S = a.S; p.Spad = a.Spad; p.D = a.D; p.Sp = Sp; p.bh0 = bh0;
        if (launch_plain(simt_apply_kernel<T, OutT, false, true>, dim3(NT * ((a.D + GT - 1) / GT), n, 1), dim3(GTHREADS), 0, st, p) != cudaSuccess)
            return MLSTM_E_CUDA;
    }
    return MLSTM_OK;
}

template <typename T>
int bwd_launch(const SimtGemmArgs& a, const SimtGemmBwdArgs& b, cudaStream_t st) {
    const int Sp = sp_of(a.S), NT = Sp / GT, group = simt_gemm_group(a.BH, a.S), nv = (a.D + GT - 1) / GT;
    for (int bh0 = 0; bh0 < a.BH; bh0 += group) {
        const int n = a.BH - bh0 < group ? a.BH - bh0 : group;
        GateArgs g{};
        g.pr[0] = GateProblem{b.dh, b.v, b.g, a.W0, nullptr};      // dT
        g.pr[1] = GateProblem{b.q, b.k, nullptr, b.W1, nullptr};   // W / n
        g.row_rel = b.gB; g.row_ref = a.An_ref; g.col_rel = a.ga; g.col_ref = a.a_ref; g.row_lo = b.gB_lo; g.col_lo = a.ga_lo;
        g.S = a.S; g.Spad = a.Spad; g.D = a.D; g.Sp = Sp; g.bh0 = bh0;
        if (launch_plain(simt_gate_kernel<T>, dim3(NT * (NT + 1) / 2, n, 2), dim3(GTHREADS), 0, st, g) != cudaSuccess) return MLSTM_E_CUDA;
        ApplyArgs p{};
        p.dot_stride = b.dot_stride;
        p.S = a.S; p.Spad = a.Spad; p.D = a.D; p.Sp = Sp; p.bh0 = bh0;
        p.pr[0] = ApplyProblem{a.W0, b.k, b.dq, b.q, b.R};
        if (launch_plain(simt_apply_kernel<T, T, false, false>, dim3(NT * nv, n, 1), dim3(GTHREADS), 0, st, p) != cudaSuccess) return MLSTM_E_CUDA;
        p.pr[0] = ApplyProblem{a.W0, b.q, b.dk, b.k, b.dI};
        p.pr[1] = ApplyProblem{b.W1, b.dh, b.dv, nullptr, nullptr};
        if (launch_plain(simt_apply_kernel<T, T, true, false>, dim3(NT * nv, n, 2), dim3(GTHREADS), 0, st, p) != cudaSuccess) return MLSTM_E_CUDA;
    }
    return MLSTM_OK;
}

}  // namespace

// One S x S matrix per slice: slices go in groups of at most GROUP_BYTES of it.  Above MAX_S a single slice would need more
// than that; mm_simt.cu, which needs no scratch, takes those.
constexpr size_t SIMT_GROUP_BYTES = size_t{256} << 20;
constexpr int SIMT_MAX_S = 8192;

bool simt_gemm_supported(int S) { return S <= SIMT_MAX_S; }

int simt_gemm_group(int BH, int S) {
    const size_t one = static_cast<size_t>(sp_of(S)) * sp_of(S) * sizeof(float);
    const size_t n = SIMT_GROUP_BYTES / one;
    return static_cast<int>(n < 1 ? 1 : n > static_cast<size_t>(BH) ? BH : n);
}

size_t simt_gemm_fwd_bytes(int BH, int S) {
    const size_t Sp = sp_of(S);
    return simt_gemm_group(BH, S) * (Sp * Sp + Sp / GT * Sp) * sizeof(float);
}

size_t simt_gemm_matrix_bytes(int BH, int S) {
    const size_t Sp = sp_of(S);
    return simt_gemm_group(BH, S) * Sp * Sp * sizeof(float);
}

int launch_simt_gemm_fwd(const SimtGemmArgs& a, const void* q, const void* k, const void* v, const void* o, void* h, int dtype,
                         int h_dtype, cudaStream_t st) {
    const bool h32 = h_dtype == MLSTM_DT_F32;
    switch (dtype) {
        case MLSTM_DT_F32: return fwd_launch<float, float>(a, q, k, v, o, h, st);
        case MLSTM_DT_F16: return h32 ? fwd_launch<__half, float>(a, q, k, v, o, h, st) : fwd_launch<__half, __half>(a, q, k, v, o, h, st);
        case MLSTM_DT_BF16:
            return h32 ? fwd_launch<__nv_bfloat16, float>(a, q, k, v, o, h, st) : fwd_launch<__nv_bfloat16, __nv_bfloat16>(a, q, k, v, o, h, st);
    }
    return MLSTM_E_ARG;
}

int launch_simt_gemm_bwd(const SimtGemmArgs& a, const SimtGemmBwdArgs& b, int dtype, cudaStream_t st) {
    switch (dtype) {
        case MLSTM_DT_F32: return bwd_launch<float>(a, b, st);
        case MLSTM_DT_F16: return bwd_launch<__half>(a, b, st);
        case MLSTM_DT_BF16: return bwd_launch<__nv_bfloat16>(a, b, st);
    }
    return MLSTM_E_ARG;
}

}  // namespace mlstm
