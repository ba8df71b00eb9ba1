// Chunkwise forward of the mLSTM for long sequences, with an inbound / outbound state so that a
// sequence can be split into contiguous segments across GPUs.
//
// The reference has no such entry point; its only long-sequence mechanism is the inter-block carry of
// the scan path (mlstm_scan.py:143-195: per-block (C, n) states reduced over blocks).  This file
// gives that mechanism the stabiliser algebra of the parallel path: with the prefix maximum A known
// up front (gates.cu), every weight is exp(a_j - A_ref) <= 1 and the carry is a plain linear
// recurrence
//     S_{k+1} = exp(A_end(k-1) - A_end(k)) S_k + U_k,    U_k = sum_{j in block k} exp(a_j - A_end(k)) k_j v_j^T
// (S is indexed [key, value]; z is the same with v dropped: the normaliser vector).  A query t of block k
// gets   num_t = intra-block part + exp(A_end(k-1) - A_t) (q_t S_k) / sqrt(D)   and the same for b_t.
// The contributions U_k come from chunk_state.cu, the output from mode FWDC of chunk_pair.cu (mm_tc.cu for an odd number of
// tiles per block).
#include "mlstm_common.cuh"

namespace mlstm {
namespace {

constexpr size_t WS_ALIGN = 256;
inline size_t al(size_t x) { return (x + WS_ALIGN - 1) / WS_ALIGN * WS_ALIGN; }
inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

template <typename T16>
__global__ void identity_kernel(T16* ident, int D) {   // D x D
    grid_dep_wait();
    grid_dep_launch();
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx < D * D) ident[idx] = from_f32<T16>((idx / D) == (idx % D) ? 1.0f : 0.0f);
}

// One thread owns four consecutive elements of a slice's state (D x D matrix and D-vector, the normaliser) and walks
// the blocks in order.  It writes the INBOUND state of every block (16-bit matrix for the tensor cores, fp32 vector;
// skipped when `states` is null) and, optionally, the state after the last block (S_end / z_end with per-slice
// strides, so that they can sit inside a packed record).
// Work split: a CTA owns 512 elements of the matrix: whole rows when only the row-major copy is written; when a
// transposed copy is wanted too, a patch of 32 rows x 16 columns (thread t: row t / 4, columns 4 (t % 4) .. +3), so
// that it writes 32 bytes per row of the row-major copy and, through a transpose in shared memory, 64 bytes per row of
// the transposed copy (written element by element from registers, the
// transposed copy cost 16 times its size in memory transactions: 0.4 ms per scan at 256 blocks of 128 x 128).
// The CTAs behind the patches own the vector.
// late_bound (optional, per slice): a carry that became known after the gate pass, see PassParams;
// block contributions U_k were stabilised by the local block-end maximum and are rescaled to the
// later, larger one on the way in.
// statesT (optional): the same per-block matrices transposed ([value, key]), for passes whose state step
// contracts over the value dimension.  reverse: walk the blocks from the last to the first, which turns
// the same recurrence into the backward's carried state R_{k-1} = exp(A_end(k-1) - A_end(k)) R_k + P_k
// (block k then receives what the LATER blocks contribute).
constexpr int SCAN_TB = 1024;       // blocks per tile of the factor tables of state_scan_kernel
constexpr int SCAN_THREADS_S = 128;
constexpr int PATCH_ROWS = 32, PATCH_COLS = 16;

template <typename T16>
__global__ void __launch_bounds__(SCAN_THREADS_S)
state_scan_kernel(const T16* __restrict__ U, const float* __restrict__ zU, const double* __restrict__ An_bound,
                  const float* __restrict__ S_in, const float* __restrict__ z_in, T16* __restrict__ states,
                  float* __restrict__ zstate, float* __restrict__ S_end, float* __restrict__ z_end, size_t S_end_stride,
                  size_t z_end_stride, int NB, int D, const double* __restrict__ late_bound,
                  const double* __restrict__ summary, double* __restrict__ summary_dst, size_t summary_dst_stride,
                  T16* __restrict__ statesT, int reverse, int* __restrict__ zero_word) {
    grid_dep_wait();
    grid_dep_launch();
    const int bh = blockIdx.y;
    const int DD = D * D;
    // the work-item counter of the pass that follows in the same call (its launcher then needs no memset of its own)
    if (zero_word && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *zero_word = 0;
    // patch shape: 32 x 16 when a transposed copy is written, else whole rows (512 consecutive elements per CTA)
    const int pcols = statesT ? PATCH_COLS : D;
    const int prows = 4 * SCAN_THREADS_S / pcols;
    const int npc = D / pcols;
    const int npatch = (D / prows) * npc;
    if (blockIdx.x == 0 && threadIdx.x == 0 && summary_dst) {
        double* dst = reinterpret_cast<double*>(reinterpret_cast<float*>(summary_dst) + bh * summary_dst_stride);
        dst[0] = summary[2 * bh];
        dst[1] = summary[2 * bh + 1];
    }
    const bool is_vec = static_cast<int>(blockIdx.x) >= npatch;     // uniform over the CTA
    const int prow0 = (blockIdx.x / npc) * prows, pcol0 = (blockIdx.x % npc) * pcols;
    const int lrow = threadIdx.x / (pcols / 4), lcol = (threadIdx.x % (pcols / 4)) * 4;
    const int off = is_vec ? ((blockIdx.x - npatch) * SCAN_THREADS_S + threadIdx.x) * 4 : (prow0 + lrow) * D + pcol0 + lcol;
    const bool valid = !is_vec || off < D;     // threads past the end still help with the factor tables and the barriers
    const size_t per_block = is_vec ? D : DD;
    // block contributions: the matrices as the tensor-core pass wrote them, the vectors in fp32
    const float* srcz = zU + static_cast<size_t>(bh) * NB * per_block + off;
    const T16* srcU = U + static_cast<size_t>(bh) * NB * per_block + off;
    const float* init = is_vec ? z_in : S_in;
    float4 s = (init && valid) ? *reinterpret_cast<const float4*>(init + static_cast<size_t>(bh) * per_block + off)
                               : make_float4(0.f, 0.f, 0.f, 0.f);
    const double* bound = An_bound + static_cast<size_t>(bh) * (NB + 1);
    const double lb = late_bound ? late_bound[bh] : INFINITY;
    // The two factors of a block (decay of the carried state, rescaling of the block's own contribution) are the
    // same for every element: the CTA computes them once per tile of SCAN_TB blocks into shared memory (evaluated
    // per thread and block they were most of the kernel's instructions: 107 per warp and block against about 20 now).
    __shared__ float sd[SCAN_TB], sc[SCAN_TB];
    // transposed patches on their way out: [column][row], two buffers so that one barrier per block is enough
    __shared__ __align__(16) T16 tp[2][PATCH_COLS][PATCH_ROWS + 8];
    const bool transposing = statesT != nullptr && !is_vec;
    const int trow = threadIdx.x >> 3, tcol = (threadIdx.x & 7) * 4;   // this thread's piece of the transposed patch
    int tbuf = 0;
    // blocks whose contributions are fetched ahead of the serial update
    constexpr int PF = 16;
    for (int t0 = 0; t0 < NB; t0 += SCAN_TB) {
        const int tn = min(SCAN_TB, NB - t0);
        __syncthreads();   // the previous tile's factors are no longer read
        for (int j = threadIdx.x; j < tn; j += blockDim.x) {
            const int kb = reverse ? NB - 1 - (t0 + j) : t0 + j;
            const double b1 = bound[kb + 1], b0 = bound[kb];
            const double b1c = fmin(b1, lb), b0c = fmin(b0, lb);
            // exp(A_end(k-1) - A_end(k)); 0 while nothing is carried in (bound = +inf: also b1 then, in left padding)
            sd[j] = b0c == static_cast<double>(INFINITY) ? 0.0f : exp2f(static_cast<float>(b1c - b0c));
            sc[j] = b1c == b1 ? 1.0f : exp2f(static_cast<float>(b1c - b1));   // < 1: the late carry raised the block's stabiliser
        }
        __syncthreads();
        if (is_vec && !valid) continue;
        for (int k0 = 0; k0 < tn; k0 += PF) {
            float4 u[PF];
            if (is_vec) {     // (uniform over the CTA: the loads of either kind go out as one batch)
#pragma unroll
                for (int j = 0; j < PF; j++) {
                    if (k0 + j < tn) {
                        const int kb = reverse ? NB - 1 - (t0 + k0 + j) : t0 + k0 + j;
                        u[j] = __ldg(reinterpret_cast<const float4*>(srcz + static_cast<size_t>(kb) * per_block));
                    }
                }
            } else {
                uint2 raw[PF];
#pragma unroll
                for (int j = 0; j < PF; j++) {
                    if (k0 + j < tn) {
                        const int kb = reverse ? NB - 1 - (t0 + k0 + j) : t0 + k0 + j;
                        raw[j] = __ldg(reinterpret_cast<const uint2*>(srcU + static_cast<size_t>(kb) * per_block));
                    }
                }
#pragma unroll
                for (int j = 0; j < PF; j++) {
                    const T16* e4 = reinterpret_cast<const T16*>(&raw[j]);
                    u[j] = make_float4(to_f32<T16>(e4[0]), to_f32<T16>(e4[1]), to_f32<T16>(e4[2]), to_f32<T16>(e4[3]));
                }
            }
#pragma unroll
            for (int j = 0; j < PF; j++) {
                if (k0 + j >= tn) break;
                const int k = reverse ? NB - 1 - (t0 + k0 + j) : t0 + k0 + j;
                if (is_vec) {
                    if (zstate) *reinterpret_cast<float4*>(zstate + (static_cast<size_t>(bh) * NB + k) * D + off) = s;
                } else if (states || statesT) {
                    T16 o[4] = {from_f32<T16>(s.x), from_f32<T16>(s.y), from_f32<T16>(s.z), from_f32<T16>(s.w)};
                    if (states)
                        *reinterpret_cast<uint2*>(states + (static_cast<size_t>(bh) * NB + k) * DD + off) = *reinterpret_cast<uint2*>(o);
                    if (transposing) {   // (uniform over the CTA)
                        tp[tbuf][lcol + 0][lrow] = o[0];
                        tp[tbuf][lcol + 1][lrow] = o[1];
                        tp[tbuf][lcol + 2][lrow] = o[2];
                        tp[tbuf][lcol + 3][lrow] = o[3];
                        __syncthreads();
                        T16* dstT = statesT + (static_cast<size_t>(bh) * NB + k) * DD + static_cast<size_t>(pcol0 + trow) * D + prow0 + tcol;
                        *reinterpret_cast<uint2*>(dstT) = *reinterpret_cast<const uint2*>(&tp[tbuf][trow][tcol]);
                        tbuf ^= 1;
                    }
                }
                const float d = sd[k0 + j], c = sc[k0 + j];
                // a decay of exactly 0 (nothing carried in) must also wipe an inbound state that is not finite
                s.x = (d == 0.0f ? 0.0f : d * s.x) + c * u[j].x;
                s.y = (d == 0.0f ? 0.0f : d * s.y) + c * u[j].y;
                s.z = (d == 0.0f ? 0.0f : d * s.z) + c * u[j].z;
                s.w = (d == 0.0f ? 0.0f : d * s.w) + c * u[j].w;
            }
        }
    }
    if (!valid) return;
    float* dst = is_vec ? z_end : S_end;
    const size_t stride = is_vec ? z_end_stride : S_end_stride;
    if (dst) *reinterpret_cast<float4*>(dst + static_cast<size_t>(bh) * stride + off) = s;
}

// Sequence-parallel fold: from the gathered records of all segments (per slice: S | z | {F_end, A_end},
// every segment's state stabilised by its OWN prefix maximum and its F counted from zero) to the
// inbound state of segment `rank` and its late carry.  With F_in(g) the log-forget total before
// segment g, segment g's stabiliser in global terms is A_g - F_in(g); the inbound maximum is
// A_in = max_{g < rank} of those, S_in = sum_g exp(A_g - F_in(g) - A_in) S_g (weights <= 1), and the
// late bound handed to the kernels is -(A_in + F_in(rank)) * log2e (+inf for the first segment).
// This is the combine of the reference's scan operators (mlstm_scan.py:15-26) over segment summaries.
__global__ void sp_fold_kernel(const float* __restrict__ gathered, int rank, int BH, int D, size_t rec_stride,
                               float* __restrict__ S_in, float* __restrict__ z_in, double* __restrict__ late_bound,
                               double* __restrict__ carry) {
    grid_dep_wait();
    grid_dep_launch();
    const int bh = blockIdx.y;
    const int DD = D * D;
    const int e = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (e >= DD + D) return;
    auto rec = [&](int g) { return gathered + (static_cast<size_t>(g) * BH + bh) * rec_stride; };
    auto tail = [&](int g) { return reinterpret_cast<const double*>(rec(g) + DD + D); };
    double Fin = 0.0, Ain = -INFINITY;
    for (int g = 0; g < rank; g++) {
        const double* t = tail(g);
        Ain = fmax(Ain, t[1] - Fin);
        Fin += t[0];
    }
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    double Fg = 0.0;
    for (int g = 0; g < rank; g++) {
        const double* t = tail(g);
        const float w = static_cast<float>(exp(t[1] - Fg - Ain));
        Fg += t[0];
        const float4 x = __ldg(reinterpret_cast<const float4*>(rec(g) + e));
        acc.x = fmaf(w, x.x, acc.x); acc.y = fmaf(w, x.y, acc.y); acc.z = fmaf(w, x.z, acc.z); acc.w = fmaf(w, x.w, acc.w);
    }
    if (e >= DD) *reinterpret_cast<float4*>(z_in + static_cast<size_t>(bh) * D + (e - DD)) = acc;
    else *reinterpret_cast<float4*>(S_in + static_cast<size_t>(bh) * DD + e) = acc;
    if (e == 0) {
        late_bound[bh] = rank == 0 ? static_cast<double>(INFINITY) : -(Ain + Fin) * 1.4426950408889634;
        if (carry) {
            carry[2 * bh] = Fin;
            carry[2 * bh + 1] = Ain;
        }
    }
}

struct ChunkWs {
    int* status;
    float *ga, *gAn, *gaw, *m, *b, *zU, *zstate, *S_in, *z_in;
    void* U;          // per-block contributions to the state, 16-bit
    double *a_ref, *An_ref, *An_bound, *gscratch, *summary, *late;
    void *ident, *states;
    int NB;
    size_t bytes;
};

// parts: 16-bit matrices a carried state is held in.  2: written by launch_carried_states, and what only the stages of
// the 1-part form use is left out; states of `group` slices at a time (0: all), m and b are the caller's
ChunkWs carve(void* ws, int BH, int S, int D, int chunk, int parts = 1, int group = 0) {
    ChunkWs w{};
    uint8_t* base = static_cast<uint8_t*>(ws);
    size_t off = 0;
    auto take = [&](size_t bytes) {
        void* p = base ? base + off : nullptr;
        off += al(bytes);
        return p;
    };
    const size_t Spad = round_up(S, TILE);
    const size_t vec = static_cast<size_t>(BH) * Spad * sizeof(float);
    w.NB = (S + chunk - 1) / chunk;
    const size_t nblk = static_cast<size_t>(group ? group : BH) * w.NB;
    w.status = static_cast<int*>(take(WS_ALIGN));
    w.ga = static_cast<float*>(take(vec));
    w.gAn = static_cast<float*>(take(vec));
    w.gaw = static_cast<float*>(take(vec));
    w.a_ref = static_cast<double*>(take(vec / REF_BLOCK * 2));
    w.An_ref = static_cast<double*>(take(vec / REF_BLOCK * 2));
    if (parts == 1) {
        w.m = static_cast<float*>(take(static_cast<size_t>(BH) * S * sizeof(float)));
        w.b = static_cast<float*>(take(static_cast<size_t>(BH) * S * sizeof(float)));
    }
    w.An_bound = static_cast<double*>(take(static_cast<size_t>(BH) * (w.NB + 1) * sizeof(double)));
    const size_t gs = gates_scratch_bytes(BH, static_cast<int>(Spad));
    w.gscratch = gs ? static_cast<double*>(take(gs)) : nullptr;
    if (parts == 1) {
        w.ident = take(static_cast<size_t>(D) * D * 2);
        w.U = take(nblk * D * D * 2);
        w.zU = static_cast<float*>(take(nblk * D * sizeof(float)));
    }
    w.states = take(nblk * D * D * 2 * parts);
    w.zstate = static_cast<float*>(take(nblk * D * sizeof(float)));
    if (parts == 1) {
        // sequence-parallel stages: this segment's gate summary, the folded inbound state and the late carry
        w.summary = static_cast<double*>(take(static_cast<size_t>(BH) * 2 * sizeof(double)));
        w.late = static_cast<double*>(take(static_cast<size_t>(BH) * sizeof(double)));
        w.S_in = static_cast<float*>(take(static_cast<size_t>(BH) * D * D * sizeof(float)));
        w.z_in = static_cast<float*>(take(static_cast<size_t>(BH) * D * sizeof(float)));
    }
    w.bytes = off;
    return w;
}

// the same workspace as the slices from bh0 on see it; the states are those of whatever group is being worked on
ChunkWs from_slice(ChunkWs w, int bh0, int S) {
    const size_t Spad = round_up(S, TILE), vec = bh0 * Spad, ref = bh0 * (Spad / REF_BLOCK), row = static_cast<size_t>(bh0) * S;
    w.ga += vec; w.gAn += vec; w.gaw += vec;
    w.a_ref += ref; w.An_ref += ref;
    w.An_bound += static_cast<size_t>(bh0) * (w.NB + 1);
    if (w.m) w.m += row;
    if (w.b) w.b += row;
    return w;
}

int check_chunk_args(int B, int NH, int S, int D, int dtype, int chunk) {
    if (B <= 0 || NH <= 0 || S <= 0 || D <= 0 || chunk <= 0) return MLSTM_E_ARG;
    if (dtype != MLSTM_DT_F16 && dtype != MLSTM_DT_BF16) return MLSTM_E_UNSUPPORTED;  // tensor-core path only
    if (D != 128 && D != 256) return MLSTM_E_UNSUPPORTED;
    if (chunk % TILE != 0) return MLSTM_E_SHAPE;
    if (static_cast<long long>(B) * NH > 65535) return MLSTM_E_SHAPE;
    return MLSTM_OK;
}

// arguments of the forward's states (chunk_state.cu): X = K, Y = V, and z, the same with V dropped
BlockStateArgs forward_states(const void* k, const void* v, const ChunkWs& w, int BH, int S, int Spad, int chunk) {
    BlockStateArgs a{};
    a.X = k; a.Y = v; a.col_w = w.gaw; a.col_ref = w.a_ref; a.An_bound = w.An_bound;
    a.S = S; a.Spad = Spad; a.BH = BH; a.NB = w.NB; a.chunk = chunk; a.status = w.status;
    a.U = w.U; a.vec = w.zU;
    return a;
}

// h of the segment from the per-block inbound states (FWDC pass)
int launch_fwdc(const void* q, const void* k, const void* v, const void* o, void* h, int h_dtype, const ChunkWs& w, int BH,
                int S, int Spad, int D, int dtype, int chunk, const double* late_bound, cudaStream_t st, int parts = 1) {
    PassParams p{};
    p.S = S; p.Spad = Spad; p.BH = BH; p.D = D; p.status = w.status; p.sched = w.status + 8;
    p.sched_zeroed = 1;   // by the state scan in front of this pass
    p.X = q; p.Y = k; p.Z = v;
    p.row_rel = w.gAn; p.row_ref = w.An_ref; p.col_rel = w.ga; p.col_w = w.gaw; p.col_ref = w.a_ref;
    p.er_add = -0.5f * log2f(static_cast<float>(D));
    p.out = h; p.m = w.m; p.b_out = w.b; p.ogate = o;
    p.chunk_tiles = chunk / TILE; p.NB = w.NB; p.An_bound = w.An_bound; p.ident = w.ident;
    p.states = w.states; p.zstate = w.zstate;
    p.late_bound = late_bound;
    p.state_parts = parts;
    if (chunk_pair_supported(D, dtype, p.chunk_tiles)) return launch_chunk_pair(FWDC, p, dtype, h_dtype, st);
    return launch_pass_tc(FWDC, p, dtype, h_dtype, st);
}

}  // namespace

int launch_identity(void* ident, int D, int dtype, cudaStream_t st) {
    const int n = D * D;
    cudaError_t ce;
    if (dtype == MLSTM_DT_BF16)
        ce = launch_plain(identity_kernel<__nv_bfloat16>, dim3((n + 255) / 256), dim3(256), 0, st, static_cast<__nv_bfloat16*>(ident), D);
    else
        ce = launch_plain(identity_kernel<__half>, dim3((n + 255) / 256), dim3(256), 0, st, static_cast<__half*>(ident), D);
    return ce == cudaSuccess ? MLSTM_OK : MLSTM_E_CUDA;
}

int launch_state_scan(const void* U, const float* zU, const double* An_bound, const float* S_in, const float* z_in,
                      void* states16, float* zstate, float* S_end, float* z_end, int BH, int NB, int D, int dtype,
                      cudaStream_t st, const double* late_bound, float* rec, size_t rec_stride, const double* summary,
                      void* statesT16, int reverse, int* zero_word) {
    // small CTAs: a slice has about 4 K threads of work, which should spread over all SMs
    const int threads = SCAN_THREADS_S;
    if (D % PATCH_ROWS != 0 || D > 4 * threads) return MLSTM_E_SHAPE;
    const int npatch = D * D / (4 * threads);
    dim3 grid(npatch + (D / 4 + threads - 1) / threads, BH);
    size_t s_stride = static_cast<size_t>(D) * D, z_stride = D;
    double* sum_dst = nullptr;
    if (rec) {   // S_end | z_end | summary inside per-slice records
        S_end = rec;
        z_end = rec + s_stride;
        sum_dst = reinterpret_cast<double*>(rec + s_stride + D);
        s_stride = z_stride = rec_stride;
    }
    cudaError_t ce;
    if (dtype == MLSTM_DT_BF16)
        ce = launch_plain(state_scan_kernel<__nv_bfloat16>, grid, dim3(threads), 0, st, static_cast<const __nv_bfloat16*>(U), zU, An_bound, S_in, z_in,
                        static_cast<__nv_bfloat16*>(states16), zstate, S_end, z_end, s_stride, z_stride, NB, D, late_bound, summary,
                        sum_dst, rec_stride, static_cast<__nv_bfloat16*>(statesT16), reverse, zero_word);
    else
        ce = launch_plain(state_scan_kernel<__half>, grid, dim3(threads), 0, st, static_cast<const __half*>(U), zU, An_bound, S_in, z_in,
                        static_cast<__half*>(states16), zstate, S_end, z_end, s_stride, z_stride, NB, D, late_bound, summary, sum_dst,
                        rec_stride, static_cast<__half*>(statesT16), reverse, zero_word);
    if (ce != cudaSuccess) return MLSTM_E_CUDA;
    return cudaGetLastError() == cudaSuccess ? MLSTM_OK : MLSTM_E_CUDA;
}

}  // namespace mlstm

using namespace mlstm;

extern "C" {

size_t mlstm_chunk_workspace(int B, int NH, int S, int D, int dtype, int chunk) {
    if (check_chunk_args(B, NH, S, D, dtype, chunk) != MLSTM_OK) return 0;
    return carve(nullptr, B * NH, S, D, chunk).bytes;
}

int mlstm_chunk_gate_summary(const void* f, const void* i, double* summary, void* workspace, size_t workspace_bytes, int B,
                             int NH, int S, int D, int dtype, int chunk, void* stream) {
    if (!f || !i || !summary) return MLSTM_E_ARG;
    int rc = check_chunk_args(B, NH, S, D, dtype, chunk);
    if (rc != MLSTM_OK) return rc;
    ChunkWs w = carve(workspace, B * NH, S, D, chunk);
    if (!workspace || workspace_bytes < w.bytes) return MLSTM_E_WORKSPACE;
    return launch_gates_fwd(f, i, nullptr, nullptr, nullptr, nullptr, nullptr, B * NH, S, round_up(S, TILE), dtype,
                            static_cast<cudaStream_t>(stream), nullptr, summary, nullptr, 0, w.gscratch);
}

int mlstm_chunk_prepare(const void* k, const void* v, const void* f, const void* i, const double* carry_in,
                        double* summary_out, void* workspace, size_t workspace_bytes, int B, int NH, int S, int D,
                        int dtype, int chunk, void* stream) {
    if (!k || !v || !f || !i) return MLSTM_E_ARG;
    int rc = check_chunk_args(B, NH, S, D, dtype, chunk);
    if (rc != MLSTM_OK) return rc;
    if (!aligned16(k) || !aligned16(v)) return MLSTM_E_ALIGN;
    const int BH = B * NH, Spad = round_up(S, TILE);
    ChunkWs w = carve(workspace, BH, S, D, chunk);
    if (!workspace || workspace_bytes < w.bytes || !aligned16(workspace)) return MLSTM_E_WORKSPACE;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // (the gate pass also clears the status word and the work-item counters)
    if ((rc = launch_gates_fwd(f, i, w.ga, w.gAn, w.a_ref, w.An_ref, w.m, BH, S, Spad, dtype, st, carry_in, summary_out,
                               w.An_bound, chunk, w.gscratch, w.gaw, w.status, STATUS_WORDS)) != MLSTM_OK)
        return rc;
    if (!chunk_pair_supported(D, dtype, chunk / TILE) && (rc = launch_identity(w.ident, D, dtype, st)) != MLSTM_OK) return rc;
    return launch_block_states(forward_states(k, v, w, BH, S, Spad, chunk), D, dtype, st);
}

int mlstm_chunk_local_state(void* workspace, size_t workspace_bytes, float* S_end, float* z_end, int B, int NH, int S,
                            int D, int dtype, int chunk, void* stream) {
    if (!S_end || !z_end) return MLSTM_E_ARG;
    int rc = check_chunk_args(B, NH, S, D, dtype, chunk);
    if (rc != MLSTM_OK) return rc;
    ChunkWs w = carve(workspace, B * NH, S, D, chunk);
    if (!workspace || workspace_bytes < w.bytes) return MLSTM_E_WORKSPACE;
    // the recurrence is linear: the state this segment adds is the scan from a zero state, with the
    // first decay taken from the carried-in stabiliser (a zero state makes that decay irrelevant)
    return launch_state_scan(w.U, w.zU, w.An_bound, nullptr, nullptr, w.states, w.zstate, S_end, z_end, B * NH, w.NB, D,
                             dtype, static_cast<cudaStream_t>(stream));
}

int mlstm_chunk_apply(const void* q, const void* k, const void* v, const void* o, const float* S_in, const float* z_in,
                      void* h, int h_dtype, float* S_out, float* z_out, void* workspace, size_t workspace_bytes, int B,
                      int NH, int S, int D, int dtype, int chunk, void* stream) {
    if (!q || !k || !v || !h) return MLSTM_E_ARG;
    if ((S_in == nullptr) != (z_in == nullptr)) return MLSTM_E_ARG;
    int rc = check_chunk_args(B, NH, S, D, dtype, chunk);
    if (rc != MLSTM_OK) return rc;
    if (h_dtype != MLSTM_DT_F32 && h_dtype != dtype) return MLSTM_E_ARG;
    if (!aligned16(q) || !aligned16(k) || !aligned16(v) || !aligned16(o) || !aligned16(h) || !aligned16(S_in) ||
        !aligned16(z_in))
        return MLSTM_E_ALIGN;
    const int BH = B * NH, Spad = round_up(S, TILE);
    ChunkWs w = carve(workspace, BH, S, D, chunk);
    if (!workspace || workspace_bytes < w.bytes) return MLSTM_E_WORKSPACE;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // (the scan also clears the work-item counter of the output pass)
    if ((rc = launch_state_scan(w.U, w.zU, w.An_bound, S_in, z_in, w.states, w.zstate, S_out, z_out, BH, w.NB, D, dtype,
                                st, nullptr, nullptr, 0, nullptr, nullptr, 0, w.status + 8 + FWDC)) != MLSTM_OK)
        return rc;
    return launch_fwdc(q, k, v, o, h, h_dtype, w, BH, S, Spad, D, dtype, chunk, nullptr, st);
}

// ------------------------------------------------------------------------------------------------
// Backward of the chunkwise forward (no inbound state): dq, dk, dv, df, di in time linear in S.
// Within a block the three parallel backward passes run restricted to the block (modes DQC, DKC, DVC of
// the tensor-core pass); across blocks dQ uses the forward's inbound state S_k, and dK, dV use a state
// carried BACK over the blocks,
//   R_k = sum_{t after block k} exp(A_end(k) - A_t) (scale / n_t) q_t dh_t^T   (+ the vector r_k with g_t q_t),
// built like the forward states: per-block contributions from chunk_state.cu (X = Q, Y = dH, column
// weights from the backward preparation), then the block recurrence walked in reverse.  dI and the row
// sums behind dF are row dots of the complete fp32 accumulators, as in the parallel backward
// (mlstm_matmul.py:256-316, 319-333 give the quantities; the reference has no chunkwise backward).
struct ChunkBwdWs {
    ChunkWs f;
    float *gB, *gBw, *g, *dI, *Rdot, *rvec;
    void *dh16;
    void *fstates;     // the forward's inbound states (1 part: transposed, for the one-CTA kernel)
    void *rstatesT;    // 1 part: transposed copy of the states carried back
    size_t bytes;
};
static ChunkBwdWs carve_bwd_chunk(void* ws, int BH, int S, int D, int chunk, bool need_dh16, int parts = 1, int group = 0) {
    ChunkBwdWs w{};
    w.f = carve(ws, BH, S, D, chunk, parts, group);
    uint8_t* base = static_cast<uint8_t*>(ws);
    size_t off = w.f.bytes;
    auto take = [&](size_t bytes) {
        void* p = base ? base + off : nullptr;
        off += al(bytes);
        return p;
    };
    const size_t vec = static_cast<size_t>(BH) * round_up(S, TILE) * sizeof(float);
    const size_t nblk = static_cast<size_t>(group ? group : BH) * w.f.NB;
    w.gB = static_cast<float*>(take(vec));
    w.gBw = static_cast<float*>(take(vec));
    w.g = static_cast<float*>(take(vec));
    w.dI = static_cast<float*>(take(vec * TC_DOT_PARTS));     // partial row dots, one per gate group
    w.Rdot = static_cast<float*>(take(vec * TC_DOT_PARTS));
    w.rvec = static_cast<float*>(take(nblk * D * sizeof(float)));
    w.fstates = take(nblk * D * D * 2 * parts);
    w.rstatesT = parts == 1 ? take(nblk * D * D * 2) : nullptr;
    w.dh16 = need_dh16 ? take(static_cast<size_t>(BH) * S * D * 2) : nullptr;
    w.bytes = off;
    return w;
}

size_t mlstm_chunk_bwd_workspace(int B, int NH, int S, int D, int dtype, int h_dtype, int chunk) {
    if (check_chunk_args(B, NH, S, D, dtype, chunk) != MLSTM_OK) return 0;
    return carve_bwd_chunk(nullptr, B * NH, S, D, chunk, h_dtype != dtype).bytes;
}

size_t mlstm_chunk_bwd_ogate_workspace(int B, int NH, int S, int D, int dtype, int h_dtype, int chunk) {
    if (check_chunk_args(B, NH, S, D, dtype, chunk) != MLSTM_OK) return 0;
    return carve_bwd_chunk(nullptr, B * NH, S, D, chunk, true).bytes;
}

// (arguments checked, workspace carved by the caller with the same `parts` and `group`)
static int chunk_bwd_core(const void* dh, const void* q, const void* k, const void* v, const void* f, const void* i, const void* h,
                          const float* m, const float* b, const void* o, void* d_o, void* dq, void* dk, void* dv, void* df, void* di,
                          const ChunkBwdWs& w, int BH, int S, int D, int dtype, int h_dtype, int chunk, int parts, int group,
                          cudaStream_t st) {
    const int Spad = round_up(S, TILE);
    int rc;
    // gates, as in the forward (the gate pass also clears the status word and the work-item counters)
    if ((rc = launch_gates_fwd(f, i, w.f.ga, w.f.gAn, w.f.a_ref, w.f.An_ref, nullptr, BH, S, Spad, dtype, st, nullptr, nullptr,
                               w.f.An_bound, chunk, w.f.gscratch, w.f.gaw, w.f.status, STATUS_WORDS)) != MLSTM_OK)
        return rc;
    // Two parts: every pass on CTA pairs, which read the states as they are.  One part: dQ and dK on the one-CTA kernel (its
    // state step contracts over transposed states).  df is a running sum of differences of the row dots of these two passes,
    // in which the rounding of a 16-bit state's path adds up (1 to 4 % of df at S = 16384, whatever the order): this entry
    // keeps the rounding it has always had there, and with it its results.
    const bool two = parts == 2;
    if (!two && (rc = launch_identity(w.f.ident, D, dtype, st)) != MLSTM_OK) return rc;
    for (int bh0 = 0; bh0 < BH; bh0 += group) {
        const int n = BH - bh0 < group ? BH - bh0 : group;
        const ChunkWs c = from_slice(w.f, bh0, S);
        const size_t vec = static_cast<size_t>(bh0) * Spad, at16 = static_cast<size_t>(bh0) * S * D * 2;   // (dh in 16 bits here)
        auto in = [&](const void* x) { return static_cast<const void*>(static_cast<const uint8_t*>(x) + at16); };
        auto out = [&](void* x) { return static_cast<void*>(static_cast<uint8_t*>(x) + at16); };
        const void *qs = in(q), *ks = in(k), *vs = in(v), *dhs = in(w.dh16 ? w.dh16 : dh);
        const float *gB = w.gB + vec, *gBw = w.gBw + vec, *g = w.g + vec;
        // forward states, as in the forward
        BlockStateArgs fwd = forward_states(ks, vs, c, n, S, Spad, chunk);
        if (two) {
            fwd.U = w.fstates; fwd.vec = c.zstate;
            if ((rc = launch_carried_states(fwd, D, dtype, st)) != MLSTM_OK) return rc;
        } else {
            if ((rc = launch_block_states(fwd, D, dtype, st)) != MLSTM_OK) return rc;
            if ((rc = launch_state_scan(c.U, c.zU, c.An_bound, nullptr, nullptr, nullptr, c.zstate, nullptr, nullptr, n, c.NB, D, dtype, st,
                                        nullptr, nullptr, 0, nullptr, w.fstates, 0)) != MLSTM_OK)
                return rc;
        }
        // delta = dh . h, n, db -> the backward's per-row vectors of all slices (and dh in the input type).  Here, right in front
        // of the pass that reads them: in front of the forward states it cost 5 of 466 us at NH = 8, S = 16384, D = 128
        if (bh0 == 0 && (rc = launch_bwd_prep(h, dh, b, m, w.f.gAn, w.gB, w.gBw, w.g, w.dh16, o, d_o, BH, S, Spad, D, h_dtype, dtype,
                                              st)) != MLSTM_OK)
            return rc;
        // the state carried back, R_k [key, value] and r_k: the recurrence in reverse over what every block contributes,
        // P_k = sum_t beta_t q_t dh_t^T, p_k = sum_t beta_t g_t q_t with beta_t = exp(A_end(k-1) - A_t) scale / n_t, g_t = db_t n_t
        BlockStateArgs bwd = fwd;
        bwd.X = qs; bwd.Y = dhs; bwd.col_w = gBw; bwd.col_ref = c.An_ref; bwd.col_g = g; bwd.reverse = 1;
        if (two) {
            bwd.U = c.states; bwd.vec = w.rvec;
            if ((rc = launch_carried_states(bwd, D, dtype, st)) != MLSTM_OK) return rc;
        } else {
            if ((rc = launch_block_states(bwd, D, dtype, st)) != MLSTM_OK) return rc;
            if ((rc = launch_state_scan(c.U, c.zU, c.An_bound, nullptr, nullptr, c.states, w.rvec, nullptr, nullptr, n, c.NB, D, dtype, st,
                                        nullptr, nullptr, 0, nullptr, w.rstatesT, 1)) != MLSTM_OK)
                return rc;
        }
        PassParams p{};
        p.S = S; p.Spad = Spad; p.BH = n; p.D = D; p.status = c.status; p.sched = c.status + 8; p.sched_zeroed = 1;
        p.chunk_tiles = chunk / TILE; p.NB = c.NB; p.An_bound = c.An_bound; p.ident = c.ident; p.state_parts = parts;
        p.dot_part_stride = static_cast<long long>(BH) * Spad;
        auto pass = [&](int mode, bool pair) {
            return pair ? launch_chunk_pair(mode, p, dtype, dtype, st) : launch_pass_tc(mode, p, dtype, dtype, st);
        };
        // dQ = ((dH V^T + g_r) * decay) K within the block, + beta (S_k dh + g z_k) from the inbound state
        p.X = dhs; p.Y = vs; p.Z = ks;
        p.row_rel = gB; p.row_ref = c.An_ref; p.row_g = g; p.col_rel = c.ga; p.col_w = c.gaw; p.col_ref = c.a_ref; p.col_g = nullptr;
        p.states = w.fstates; p.zstate = c.zstate;
        p.out = out(dq); p.dot_src = qs; p.dot_out = w.Rdot + vec;
        if ((rc = pass(DQC, two)) != MLSTM_OK) return rc;
        // dK = ((V dH^T + g_c) * decay) Q within the block, + gamma (R_k v + r_k) from the later blocks
        p.X = vs; p.Y = dhs; p.Z = qs;
        p.row_rel = c.ga; p.row_ref = c.a_ref; p.row_g = nullptr; p.col_rel = gB; p.col_w = gBw; p.col_ref = c.An_ref; p.col_g = g;
        p.states = two ? c.states : w.rstatesT; p.rvec = w.rvec;
        p.out = out(dk); p.dot_src = ks; p.dot_out = w.dI + vec;
        if ((rc = pass(DKC, two)) != MLSTM_OK) return rc;
        // dV = ((K Q^T) * decay / n) dH within the block, + gamma R_k^T k from the later blocks
        p.X = ks; p.Y = qs; p.Z = dhs;
        p.col_g = nullptr; p.states = c.states;
        p.out = out(dv); p.dot_src = nullptr; p.dot_out = nullptr;
        if ((rc = pass(DVC, chunk_pair_supported(D, dtype, p.chunk_tiles))) != MLSTM_OK) return rc;
    }
    return launch_df(f, w.dI, w.Rdot, df, di, BH, S, Spad, dtype, st, TC_DOT_PARTS, static_cast<long long>(BH) * Spad, w.f.gscratch);
}

static int chunk_bwd_impl(const void* dh, const void* q, const void* k, const void* v, const void* f, const void* i, const void* h,
                          const float* m, const float* b, const void* o, void* d_o, void* dq, void* dk, void* dv, void* df, void* di,
                          void* workspace, size_t workspace_bytes, int B, int NH, int S, int D, int dtype, int h_dtype, int chunk,
                          void* stream) {
    if (!dh || !q || !k || !v || !f || !i || !h || !m || !b || !dq || !dk || !dv || !df || !di) return MLSTM_E_ARG;
    int rc = check_chunk_args(B, NH, S, D, dtype, chunk);
    if (rc != MLSTM_OK) return rc;
    if (h_dtype != MLSTM_DT_F32 && h_dtype != dtype) return MLSTM_E_ARG;
    if (!aligned16(dh) || !aligned16(q) || !aligned16(k) || !aligned16(v) || !aligned16(h) || !aligned16(dq) ||
        !aligned16(dk) || !aligned16(dv))
        return MLSTM_E_ALIGN;
    // dh in the input type, taken through the output gate where there is one
    ChunkBwdWs w = carve_bwd_chunk(workspace, B * NH, S, D, chunk, o || h_dtype != dtype);
    if (!workspace || workspace_bytes < w.bytes || !aligned16(workspace)) return MLSTM_E_WORKSPACE;
    return chunk_bwd_core(dh, q, k, v, f, i, h, m, b, o, d_o, dq, dk, dv, df, di, w, B * NH, S, D, dtype, h_dtype, chunk, 1, B * NH,
                          static_cast<cudaStream_t>(stream));
}

int mlstm_chunk_bwd(const void* dh, const void* q, const void* k, const void* v, const void* f, const void* i, const void* h,
                    const float* m, const float* b, void* dq, void* dk, void* dv, void* df, void* di, void* workspace,
                    size_t workspace_bytes, int B, int NH, int S, int D, int dtype, int h_dtype, int chunk, void* stream) {
    return chunk_bwd_impl(dh, q, k, v, f, i, h, m, b, nullptr, nullptr, dq, dk, dv, df, di, workspace, workspace_bytes, B, NH, S, D,
                          dtype, h_dtype, chunk, stream);
}

int mlstm_chunk_bwd_ogate(const void* dh, const void* q, const void* k, const void* v, const void* f, const void* i, const void* h,
                          const float* m, const float* b, const void* o, void* dq, void* dk, void* dv, void* df, void* di, void* d_o,
                          void* workspace, size_t workspace_bytes, int B, int NH, int S, int D, int dtype, int h_dtype, int chunk,
                          void* stream) {
    if (!o || !d_o) return MLSTM_E_ARG;
    if (!aligned16(o) || !aligned16(d_o)) return MLSTM_E_ALIGN;
    return chunk_bwd_impl(dh, q, k, v, f, i, h, m, b, o, d_o, dq, dk, dv, df, di, workspace, workspace_bytes, B, NH, S, D, dtype,
                          h_dtype, chunk, stream);
}

int mlstm_chunk_read_mb(const void* workspace, size_t workspace_bytes, float* m, float* b, int B, int NH, int S, int D, int dtype,
                        int chunk, void* stream) {
    if (!m || !b) return MLSTM_E_ARG;
    int rc = check_chunk_args(B, NH, S, D, dtype, chunk);
    if (rc != MLSTM_OK) return rc;
    ChunkWs w = carve(const_cast<void*>(workspace), B * NH, S, D, chunk);
    if (!workspace || workspace_bytes < w.bytes) return MLSTM_E_WORKSPACE;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const size_t bytes = static_cast<size_t>(B) * NH * S * sizeof(float);
    if (cudaMemcpyAsync(m, w.m, bytes, cudaMemcpyDeviceToDevice, st) != cudaSuccess) return MLSTM_E_CUDA;
    if (cudaMemcpyAsync(b, w.b, bytes, cudaMemcpyDeviceToDevice, st) != cudaSuccess) return MLSTM_E_CUDA;
    return MLSTM_OK;
}

size_t mlstm_chunk_sp_record_floats(int D) { return D > 0 ? static_cast<size_t>(D) * D + D + 4 : 0; }

int mlstm_chunk_sp_local(const void* k, const void* v, const void* f, const void* i, float* record, void* workspace,
                         size_t workspace_bytes, int B, int NH, int S, int D, int dtype, int chunk, void* stream) {
    if (!record) return MLSTM_E_ARG;
    if (!aligned16(record)) return MLSTM_E_ALIGN;
    ChunkWs w = carve(workspace, B * NH, S, D, chunk);
    // gates and block states with no carry; this segment's own summary goes to the workspace
    int rc = mlstm_chunk_prepare(k, v, f, i, nullptr, workspace ? w.summary : nullptr, workspace, workspace_bytes, B, NH, S, D,
                                 dtype, chunk, stream);
    if (rc != MLSTM_OK) return rc;
    // the state the segment adds, stabilised by its own last prefix maximum, written into the record with the summary
    return launch_state_scan(w.U, w.zU, w.An_bound, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, B * NH, w.NB, D,
                             dtype, static_cast<cudaStream_t>(stream), nullptr, record, mlstm_chunk_sp_record_floats(D),
                             w.summary);
}

int mlstm_chunk_sp_apply(const void* q, const void* k, const void* v, const void* o, const float* gathered, int world,
                         int rank, void* h, int h_dtype, double* carry_out, void* workspace, size_t workspace_bytes, int B,
                         int NH, int S, int D, int dtype, int chunk, void* stream) {
    if (!q || !k || !v || !h || !gathered) return MLSTM_E_ARG;
    if (world <= 0 || rank < 0 || rank >= world) return MLSTM_E_ARG;
    int rc = check_chunk_args(B, NH, S, D, dtype, chunk);
    if (rc != MLSTM_OK) return rc;
    if (h_dtype != MLSTM_DT_F32 && h_dtype != dtype) return MLSTM_E_ARG;
    if (!aligned16(q) || !aligned16(k) || !aligned16(v) || !aligned16(o) || !aligned16(h) || !aligned16(gathered))
        return MLSTM_E_ALIGN;
    const int BH = B * NH, Spad = round_up(S, TILE);
    ChunkWs w = carve(workspace, BH, S, D, chunk);
    if (!workspace || workspace_bytes < w.bytes) return MLSTM_E_WORKSPACE;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    {
        const int threads = 256;
        const int work = (D * D + D) / 4;
        dim3 grid((work + threads - 1) / threads, BH);
        sp_fold_kernel<<<grid, threads, 0, st>>>(gathered, rank, BH, D, mlstm_chunk_sp_record_floats(D), w.S_in, w.z_in,
                                                 w.late, carry_out);
        if (cudaGetLastError() != cudaSuccess) return MLSTM_E_CUDA;
    }
    if ((rc = launch_state_scan(w.U, w.zU, w.An_bound, w.S_in, w.z_in, w.states, w.zstate, nullptr, nullptr, BH, w.NB, D,
                                dtype, st, w.late, nullptr, 0, nullptr, nullptr, 0, w.status + 8 + FWDC)) != MLSTM_OK)
        return rc;
    return launch_fwdc(q, k, v, o, h, h_dtype, w, BH, S, Spad, D, dtype, chunk, w.late, st);
}

}  // extern "C"

namespace mlstm {

// Blocks of 256 positions: at 512 the states cost half, but the passes inside a block wait for their gate warps (16-bit
// states, B = 16, NH = 8, S = 4096, D = 256, forward + backward: 2.64 ms at 256, 2.91 at 512, 3.31 at 1024).
constexpr int MM_CHUNK = 256;

// Where the chunkwise form beats the quadratic kernels.  It needs slices (a CTA walks a slice's blocks, 5 us each) and length:
// with few slices the walk is long, but the quadratic cost, S times the number of positions, is longer still.
// Measured bf16, us, quadratic -> chunkwise, forward | backward:
//   D = 128   BH 32: S 2048 60 -> 70 | 203 -> 190, S 4096 148 -> 121 | 506 -> 338    BH 64: S 1024 44 -> 53 | 150 -> 156,
//             S 2048 97 -> 88 | 343 -> 267    BH 128: S 1024 72 -> 74 | 250 -> 233, S 4096 596 -> 275 | 2135 -> 904
//             BH 16: S 4096 83 -> 103 | 274 -> 261, S 8192 258 -> 194 | 878 -> 489
//   D = 256   BH 32: S 2048 99 -> 101 | 284 -> 295, S 4096 221 -> 203 | 712 -> 569    BH 64: S 1024 78 -> 88 | 237 -> 261,
//             S 2048 149 -> 148 | 496 -> 458    BH 128: S 1024 139 -> 149 | 456 -> 450, S 4096 986 -> 618 | 3128 -> 1791
//             BH 16: S 4096 117 -> 140 | 375 -> 381, S 8192 375 -> 317 | 1182 -> 762
// and along the line itself, S = 131072 / BH:
//   D = 128   BH 1: 3695 -> 2220 | 12581 -> 4498, BH 2: 1876 -> 1156 | 6474 -> 2380, BH 4: 969 -> 631 | 3098 -> 1338,
//             BH 8: 516 -> 354 | 1637 -> 788, BH 24: 223 -> 178 | 684 -> 434, BH 64: 123 -> 114 | 367 -> 291
//   D = 256   BH 1: 5485 -> 2622 | 17035 -> 5373, BH 2: 2539 -> 1758 | 8995 -> 3166, BH 4: 1320 -> 937 | 4399 -> 1790,
//             BH 8: 691 -> 438 | 2141 -> 1011, BH 24: 345 -> 245 | 944 -> 692, BH 64: 171 -> 169 | 511 -> 459
// bf16 only: a state is a sum over positions, and fp16's range (65504) is too small for what the quadratic kernels add up
// in fp32.  The forced paths keep the kernels they name.
bool mm_chunk_route(int BH, int S, int D, int dtype, int flags) {
    if (flags & (MLSTM_F_FORCE_SIMT | MLSTM_F_FORCE_TC)) return false;
    if (dtype != MLSTM_DT_BF16 || (D != 128 && D != 256)) return false;
    return S >= 2048 && static_cast<long long>(BH) * S >= 131072;
}

// Slices whose states are in the workspace at one time.  A state costs 4 D bytes per position of its slice (two 16-bit
// matrices per block of 256), so slices go in groups, of about the same size: as many as fit MM_STATE_BYTES of one set of
// states, but no fewer than one wave of the states' kernel (D / 128 CTAs per slice on 148 SMs: 148 and 74 slices), because a
// CTA walks its slice however few there are beside it, and smaller groups would walk one after the other.  A set then takes
// at most MM_STATE_BYTES or 75 KB per position of the sequence, whatever the number of slices, and the groups walk in as many
// waves as all slices at once would.  One set forward, two backward (S_k and R_k).
// Measured, all slices at once -> two groups, us, forward | backward, both in turn (the runs of one side differ by 3 to 8 %):
// 96 x 32768 at D = 256 3519 - 3746 -> 3417 - 3687 | 10620 - 11106 -> 10593 - 11123, 160 x 65536 at D = 128 5621 - 6108 ->
// 5628 - 6074 | 17397 - 18643 -> 17748 - 18573.
constexpr size_t MM_STATE_BYTES = size_t{1} << 30;
constexpr int MM_WAVE_CTAS = 148;     // (a constant: the workspace query runs without a device)
static int mm_chunk_group(int BH, int S, int D) {
    const size_t one = static_cast<size_t>((S + MM_CHUNK - 1) / MM_CHUNK) * D * D * 2 * 2;
    const size_t fit = MM_STATE_BYTES / one, wave = MM_WAVE_CTAS / (D / TILE);
    const size_t most = fit > wave ? fit : wave;
    const int groups = static_cast<int>((BH + most - 1) / most);
    return (BH + groups - 1) / groups;
}

size_t mm_chunk_fwd_bytes(int BH, int S, int D) {
    return carve(nullptr, BH, S, D, MM_CHUNK, 2, mm_chunk_group(BH, S, D)).bytes;
}

int mm_chunk_fwd(const void* q, const void* k, const void* v, const void* f, const void* i, void* h, float* m, float* b, void* workspace,
                 int BH, int S, int D, int dtype, int h_dtype, cudaStream_t st) {
    const int group = mm_chunk_group(BH, S, D);
    ChunkWs w = carve(workspace, BH, S, D, MM_CHUNK, 2, group);
    w.m = m;
    w.b = b;
    const int Spad = round_up(S, TILE);
    int rc;
    // (the gate pass also clears the status word)
    if ((rc = launch_gates_fwd(f, i, w.ga, w.gAn, w.a_ref, w.An_ref, m, BH, S, Spad, dtype, st, nullptr, nullptr, w.An_bound, MM_CHUNK,
                               w.gscratch, w.gaw, w.status, STATUS_WORDS)) != MLSTM_OK)
        return rc;
    for (int bh0 = 0; bh0 < BH; bh0 += group) {
        const int n = BH - bh0 < group ? BH - bh0 : group;
        const size_t at = static_cast<size_t>(bh0) * S * D;
        auto in = [&](const void* x) { return static_cast<const void*>(static_cast<const uint8_t*>(x) + at * 2); };
        const ChunkWs c = from_slice(w, bh0, S);
        BlockStateArgs a = forward_states(in(k), in(v), c, n, S, Spad, MM_CHUNK);
        a.U = c.states; a.vec = c.zstate;
        if ((rc = launch_carried_states(a, D, dtype, st)) != MLSTM_OK) return rc;
        void* hs = static_cast<uint8_t*>(h) + at * (h_dtype == MLSTM_DT_F32 ? 4 : 2);
        if ((rc = launch_fwdc(in(q), in(k), in(v), nullptr, hs, h_dtype, c, n, S, Spad, D, dtype, MM_CHUNK, nullptr, st, 2)) != MLSTM_OK)
            return rc;
    }
    return MLSTM_OK;
}

size_t mm_chunk_bwd_bytes(int BH, int S, int D, bool dh_copy) {
    return carve_bwd_chunk(nullptr, BH, S, D, MM_CHUNK, dh_copy, 2, mm_chunk_group(BH, S, D)).bytes;
}

int mm_chunk_bwd(const void* dh, const void* q, const void* k, const void* v, const void* f, const void* i, const void* h, const float* m,
                 const float* b, const void* o, void* d_o, void* dq, void* dk, void* dv, void* df, void* di, void* workspace, int BH,
                 int S, int D, int dtype, int h_dtype, cudaStream_t st) {
    const int group = mm_chunk_group(BH, S, D);
    const ChunkBwdWs w = carve_bwd_chunk(workspace, BH, S, D, MM_CHUNK, o || h_dtype != dtype, 2, group);
    return chunk_bwd_core(dh, q, k, v, f, i, h, m, b, o, d_o, dq, dk, dv, df, di, w, BH, S, D, dtype, h_dtype, MM_CHUNK, 2, group, st);
}

}  // namespace mlstm
