// The states that the chunkwise form carries from block to block (16-bit inputs, head dimension 128 or 256; the carried form
// below for bf16 only):
//     U_k = sum_j w_j x_j y_j^T,  w_j = exp2(col_rel_j + col_ref_j + bound)          (x_j, y_j the rows of block k)
//     u_k = sum_j w_j g_j x_j                                                        (fp32; g_j = 1 in the forward)
// forward   x = K, y = V, bound = -A_end(k):      the states of mlstm_scan.py:74-137 with the stabiliser known up front
// reverse   x = Q, y = dH, bound = +A_end(k - 1): the contributions to the state the backward carries back, g = db n
// A plain contraction over the block's positions: both operands are read MN-major from shared memory, where the rows of X
// are first scaled.  The vector part rides along on the unrounded products.
//
// Two forms:
//   block_states     U_k and u_k of every block, 16-bit; chunk.cu then walks the recurrence (state_scan_kernel).  For a few
//                    long slices, whose blocks have to be spread over the chip, and for states that come in or go out.
//   carried_states   (CARRY) the recurrence S_{k+1} = exp(A_end(k-1) - A_end(k)) S_k + U_k in the same kernel: a CTA owns 128
//                    rows of one slice's state and walks the blocks, U in one half of TMEM, S in fp32 in the other, so that no
//                    contribution ever goes to memory.  What is written is the state in front of every block, as two 16-bit
//                    matrices (hi, and what hi leaves out), and the scaled rows of X enter the contraction as hi + mid as
//                    well: a carried part has fp32-level accuracy (16 bits and more), unlike in the 16-bit form.  For
//                    many slices: the parallel entry points' long sequences.
//
// What bounds it: HBM (X and Y once, the states out).  Per block and CTA at D = 256, blocks of 256: 256 KB = 10800 cycles at
// an SM's share of HBM, against 4100 cycles of tensor pipe (hi and mid).  The read-out updates S first and gives U back
// before it converts and stores: with the stores in front of that the next block's contraction waited for them (BH = 64,
// S = 4096, D = 256, carried: 128 us; now 100, 5.4 TB/s).  The D / 128 row halves of a slice run on neighbouring CTAs and
// share Y in L2.  Slots of 64 positions.  With few slices it is latency, 5 us per block of 256 (BH = 32, D = 128): see the
// rule in chunk.cu for where the carried form is used.  block_states took the place of a pass that brought K through an
// identity into TMEM to transpose it (S = 65536, NH = 8, D = 128: forward 325 -> 301 us together with the output pass on
// pairs; S = 16384, training step: 477 -> 462).
#include <atomic>

#include "mlstm_common.cuh"
#include "ptx_sm100.cuh"
#include "tc_host.cuh"

namespace mlstm {
namespace {

using namespace ptx;

constexpr int PB = 64;                          // positions per slot (one reference block of the gate vectors)
static_assert(PB == REF_BLOCK, "one column reference per slot");
constexpr int EPI_WARPS = 8, SCALE_WARPS = 8;   // read-out: two warps per TMEM lane quarter; scaling: 16 columns of X per warp
constexpr int NTHREADS_ST = 32 * (4 + EPI_WARPS + SCALE_WARPS);   // producer, MMA issuer, two idle warps, read-out, scaling
constexpr long long WAIT_LIMIT_ST = 4000000000LL;
constexpr float MAX_EXP2 = 60.0f;               // a reference block of pure padding has no reference of its own (its factors are 0)
constexpr int SLEEP_NS_ST = 32;
constexpr int GROUP_BYTES = PB * 128;           // one 128-byte column group of a slot

// decay of a state over a block from its boundaries' -A*log2e; nothing carried in (+inf) decays to nothing, also where the
// block has no finite position of its own (input gates of -inf: left padding)
__device__ __forceinline__ float block_decay(double b0, double b1) {
    return b0 == static_cast<double>(INFINITY) ? 0.0f : exp2f(static_cast<float>(b1 - b0));
}

template <int D, bool CARRY>
struct StCfg {
    static constexpr int X_BYTES = PB * TILE * 2;               // 64 positions x 128 columns of X
    static constexpr int XPARTS = CARRY ? 2 : 1;                // scaled X: hi, mid
    static constexpr int Y_BYTES = PB * D * 2;
    static constexpr int LOAD_BYTES = X_BYTES + Y_BYTES;
    static constexpr int SLOT = XPARTS * X_BYTES + Y_BYTES;     // X | (X mid) | Y
    static constexpr int NSLOT = 196608 / SLOT;
    static constexpr int STAGE = CARRY ? 4096 : 2048;           // per read-out warp: 32 rows x 32 columns (hi | mid)
    static constexpr int NACC = CARRY ? 1 : 2;                  // accumulators (CARRY: the other half of TMEM is S)
    static constexpr int NBAR = 3 * NSLOT + 2 * NACC;
    static constexpr int SMEM = NSLOT * SLOT + EPI_WARPS * STAGE + NBAR * 8 + 16;
    static_assert(SMEM <= 232448, "exceeds the shared memory of a CTA");
};

template <int D, int ABFMT, bool CARRY>
__global__ void __launch_bounds__(NTHREADS_ST, 1)
states_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmY,
              const __grid_constant__ CUtensorMap tmU, const BlockStateArgs p) {
    using C = StCfg<D, CARRY>;
    constexpr int NHV = D / TILE;                // row halves of a state
    // two values as one register of 16-bit ones, and back
    auto pack2 = [](float a, float b) {
        if constexpr (ABFMT == 1) {
            const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
            return *reinterpret_cast<const uint32_t*>(&v);
        } else {
            const __half2 v = __floats2half2_rn(a, b);
            return *reinterpret_cast<const uint32_t*>(&v);
        }
    };
    auto unpack2 = [](uint32_t x) {
        if constexpr (ABFMT == 1) return make_float2(__uint_as_float(x << 16), __uint_as_float(x & 0xffff0000u));
        else return __half22float2(*reinterpret_cast<const __half2*>(&x));
    };
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sStage = smem + C::NSLOT * C::SLOT;
    uint64_t* bar_full = reinterpret_cast<uint64_t*>(sStage + EPI_WARPS * C::STAGE);   // [NSLOT] loaded
    uint64_t* bar_scaled = bar_full + C::NSLOT;      // [NSLOT] X scaled (one arrival per scaling warp)
    uint64_t* bar_empty = bar_scaled + C::NSLOT;     // [NSLOT] no longer read by MMAs
    uint64_t* bar_acc = bar_empty + C::NSLOT;        // [NACC] U complete
    uint64_t* bar_accfree = bar_acc + C::NACC;       // [NACC] U read out (one arrival per read-out warp)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_full + C::NBAR);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // One block of one item.  CARRY: an item is 128 rows of a slice's state, its blocks come in order (step 0 first) and the
    // last one only receives; else an item is 128 rows of one block's U.
    struct Block {
        int bh, half, blk, step, t0, nslots;
    };
    auto for_blocks = [&](auto&& fn) {
        const int total = NHV * p.BH * (CARRY ? 1 : p.NB);
        for (int id = blockIdx.x; id < total; id += gridDim.x) {
            Block b;
            b.half = id % NHV;
            const int w = id / NHV;
            b.bh = CARRY ? w : w / p.NB;
            for (int j = 0; j < (CARRY ? p.NB : 1); j++) {
                b.blk = CARRY ? (p.reverse ? p.NB - 1 - j : j) : w - b.bh * p.NB;
                b.step = j;
                b.t0 = b.blk * p.chunk;
                b.nslots = (min(p.chunk, p.S - b.t0) + PB - 1) / PB;   // at least one
                if (!fn(b)) return;
            }
        }
    };
    auto contributes = [&](const Block& b) { return !CARRY || b.step < p.NB - 1; };
    if (threadIdx.x == 0) {
        for (int s = 0; s < C::NSLOT; s++) {
            mbar_init(&bar_full[s], 1);
            mbar_init(&bar_scaled[s], SCALE_WARPS);
            mbar_init(&bar_empty[s], 1);
        }
        for (int s = 0; s < C::NACC; s++) {
            mbar_init(&bar_acc[s], 1);
            mbar_init(&bar_accfree[s], EPI_WARPS);
        }
        *abort_flag = (smem_u32(smem) & 1023u) != 0;     // the swizzled tiles need a 1024-byte aligned base; never seen
        fence_mbar_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, 2 * D);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tmem_U = tmem_base + (CARRY ? D : 0);
    grid_dep_wait();      // nothing above touched global memory
    grid_dep_launch();

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer
        if (lane == 0) {
            prefetch_tmap(&tmX);
            prefetch_tmap(&tmY);
            int seq = 0;
            for_blocks([&](const Block& b) {
                if (!contributes(b)) return true;
                for (int c = 0; c < b.nslots; c++, seq++) {
                    const int s = seq % C::NSLOT;
                    if (!mbar_wait<SLEEP_NS_ST>(&bar_empty[s], ((seq / C::NSLOT) & 1) ^ 1, abort_flag, WAIT_LIMIT_ST)) return false;
                    mbar_expect_tx(&bar_full[s], C::LOAD_BYTES);
                    uint8_t* dst = smem + s * C::SLOT;
                    tma_load_4d(dst, &tmX, &bar_full[s], 0, b.t0 + c * PB, b.half * 2, b.bh);     // rows past S read as zeros
                    tma_load_4d(dst + C::XPARTS * C::X_BYTES, &tmY, &bar_full[s], 0, b.t0 + c * PB, 0, b.bh);
                }
                return true;
            });
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer (whole warp, one elected lane issues)
        const bool issuer = elect_one();
        auto uni = [](int x) { return __shfl_sync(0xffffffffu, x, 0); };
        constexpr uint32_t idesc = make_idesc(ABFMT, 128, D, 1, 1);
        const uint32_t smem_u = static_cast<uint32_t>(uni(static_cast<int>(smem_u32(smem))));
        const uint32_t tmem_u = static_cast<uint32_t>(uni(static_cast<int>(tmem_U)));
        const uint64_t xdesc0 = smem_desc_sw128(smem_u, GROUP_BYTES, 1024, 2);
        const uint64_t ydesc0 = smem_desc_sw128(smem_u + C::XPARTS * C::X_BYTES, GROUP_BYTES, 1024, 2);
        int seq = 0, n = 0;
        for_blocks([&](const Block& b) {
            if (!contributes(b)) return true;
            const int buf = n % C::NACC;
            if (!mbar_wait_warp(&bar_accfree[buf], ((n / C::NACC) & 1) ^ 1, abort_flag, WAIT_LIMIT_ST)) return false;
            tc_fence_after();
            for (int c = 0; c < b.nslots; c++, seq++) {
                const int s = seq % C::NSLOT;
                const uint32_t par = (seq / C::NSLOT) & 1;
                if (!mbar_wait_warp(&bar_full[s], par, abort_flag, WAIT_LIMIT_ST)) return false;
                if (!mbar_wait_warp(&bar_scaled[s], par, abort_flag, WAIT_LIMIT_ST)) return false;
                tc_fence_after();
                const uint64_t xd = smem_desc_advance(xdesc0, s * C::SLOT), yd = smem_desc_advance(ydesc0, s * C::SLOT);
                if (issuer) {
#pragma unroll
                    for (int part = 0; part < C::XPARTS; part++)
#pragma unroll
                        for (int kk = 0; kk < PB / 16; kk++)
                            mma_ss<false>(tmem_u + buf * D, smem_desc_advance(xd, part * C::X_BYTES + kk * 2048),
                                          smem_desc_advance(yd, kk * 2048), idesc, (c > 0 || part > 0 || kk > 0) ? 1u : 0u);
                    tc_commit(&bar_empty[s]);
                    if (c == b.nslots - 1) tc_commit(&bar_acc[buf]);
                }
                __syncwarp();
            }
            n++;
            return true;
        });
    } else if (warp >= 4 && warp < 4 + EPI_WARPS) {
        // ------------------------------------------------------------ read-out, through staging and TMA stores
        if (lane == 0) prefetch_tmap(&tmU);
        const int q32 = (warp & 3) * 32;
        constexpr int COLS = D / 2;                                  // this warp's columns
        const int c0 = ((warp - 4) >> 2) * COLS;
        const uint32_t lane_bits = static_cast<uint32_t>(q32) << 16;
        uint8_t* stage = sStage + (warp - 4) * C::STAGE;
        const int sw = (lane >> 1) & 3;                              // the 64-byte swizzle of the output map
        auto stage_row = [&](int part, const uint32_t (&o)[16]) {
#pragma unroll
            for (int j = 0; j < 4; j++)
                *reinterpret_cast<uint4*>(stage + part * 2048 + lane * 64 + ((j ^ sw) << 4)) =
                    make_uint4(o[4 * j], o[4 * j + 1], o[4 * j + 2], o[4 * j + 3]);
        };
        int n = 0;                                                   // blocks' U read out so far
        float decay = 0.0f;                                          // CARRY: of the block before
        for_blocks([&](const Block& b) {
            const int buf = n % C::NACC;
            const bool have_u = !CARRY || b.step > 0;
            if (have_u) {
                if (!mbar_wait_warp<SLEEP_NS_ST>(&bar_acc[buf], (n / C::NACC) & 1, abort_flag, WAIT_LIMIT_ST)) return false;
                tc_fence_after();
            }
            const int z = (b.bh * p.NB + b.blk) * C::XPARTS;
            auto release = [&]() {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&bar_accfree[buf]);
            };
            const uint32_t tmem_S = tmem_base + lane_bits + c0;
            if constexpr (CARRY) {
                // S = decay S + U first, so that the next block's contraction waits for this and not for the stores
                if (b.step > 0) {
                    const bool fresh = b.step == 1 || decay == 0.0f;  // (a decay of exactly 0 wipes the state, whatever it holds)
#pragma unroll 1
                    for (int ch = 0; ch < COLS / 32; ch++) {
                        uint32_t uv[32];
                        tmem_ld32(tmem_U + lane_bits + c0 + ch * 32, uv);
                        if (!fresh) {
                            uint32_t sv[32];
                            tmem_ld32(tmem_S + ch * 32, sv);
                            tc_wait_ld();
#pragma unroll
                            for (int j = 0; j < 32; j++) uv[j] = __float_as_uint(fmaf(decay, __uint_as_float(sv[j]), __uint_as_float(uv[j])));
                        } else {
                            tc_wait_ld();
                        }
                        tmem_st32(tmem_S + ch * 32, uv);
                    }
                    tc_wait_st();
                    release();
                }
            }
#pragma unroll 1
            for (int ch = 0; ch < COLS / 32; ch++) {
                uint32_t x[32];
                if (have_u) {
                    tmem_ld32(CARRY ? tmem_S + ch * 32 : tmem_U + lane_bits + buf * D + c0 + ch * 32, x);
                    tc_wait_ld();
                } else {
#pragma unroll
                    for (int j = 0; j < 32; j++) x[j] = 0u;
                }
                if (!CARRY && ch == COLS / 32 - 1) release();
                uint32_t hi[16];
                [[maybe_unused]] uint32_t mid[16];
#pragma unroll
                for (int j = 0; j < 16; j++) {
                    const float x0 = __uint_as_float(x[2 * j]), x1 = __uint_as_float(x[2 * j + 1]);
                    hi[j] = pack2(x0, x1);
                    if constexpr (CARRY) {
                        const float2 h2 = unpack2(hi[j]);
                        mid[j] = pack2(x0 - h2.x, x1 - h2.y);
                    }
                }
                if (lane == 0) bulk_wait_read_all();     // the previous stores have read the staging rows
                __syncwarp();
                stage_row(0, hi);
                if constexpr (CARRY) stage_row(1, mid);
                fence_async_smem();
                __syncwarp();
                if (lane == 0) {
#pragma unroll
                    for (int part = 0; part < C::XPARTS; part++)
                        tma_store_3d(&tmU, stage + part * 2048, c0 + ch * 32, b.half * TILE + q32, z + part);
                    bulk_commit();
                }
            }
            if (have_u) n++;
            if constexpr (CARRY) {
                const double* bound = p.An_bound + static_cast<size_t>(b.bh) * (p.NB + 1) + b.blk;
                decay = block_decay(bound[0], bound[1]);
            }
            return true;
        });
        if (lane == 0) bulk_wait_all();
        tc_fence_before();
    } else if (warp >= 4 + EPI_WARPS) {
        // ------------------------------------------------------------ scaling warps: 16 columns of X each, rows lane and lane + 32
        const int sw_warp = warp - 4 - EPI_WARPS;
        const int r7 = lane & 7;
        // byte offset of this thread's two 16-byte pieces inside a row of its column group (128-byte swizzle)
        const int group = sw_warp >> 2, piece = (sw_warp & 3) * 2;
        const int off0 = group * GROUP_BYTES + lane * 128 + ((piece ^ r7) << 4);
        const int off1 = group * GROUP_BYTES + lane * 128 + (((piece + 1) ^ r7) << 4);
        // after the reduction at a block's end lane l holds column my_col (both lanes of a pair the same)
        const int my_col = sw_warp * 16 + ((lane >> 4) & 1) * 8 + ((lane >> 3) & 1) * 4 + ((lane >> 2) & 1) * 2 + ((lane >> 1) & 1);
        int seq = 0;
        float zrun = 0.0f;
        for_blocks([&](const Block& b) {
            const double* bound = p.An_bound + static_cast<size_t>(b.bh) * (p.NB + 1) + b.blk;
            const size_t out = (static_cast<size_t>(b.bh) * p.NB + b.blk) * D + b.half * TILE + my_col;
            if (CARRY) {
                if (b.step == 0) zrun = 0.0f;
                if ((lane & 1) == 0) p.vec[out] = zrun;
                if (!contributes(b)) return true;
            }
            const double b0 = bound[0], b1 = bound[1];
            const double bnd = p.reverse ? -b0 : b1;
            float z[16];
#pragma unroll
            for (int k = 0; k < 16; k++) z[k] = 0.0f;
            // what a slot needs from the gate vectors is requested before the wait for the slot
            const size_t cols = static_cast<size_t>(b.bh) * p.Spad + b.t0 + lane;
            const double* refs = p.col_ref + static_cast<size_t>(b.bh) * (p.Spad / REF_BLOCK) + b.t0 / REF_BLOCK;
            float wn[2], gn[2] = {1.0f, 1.0f};
            double rn;
            auto load_cols = [&](int c) {
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    wn[k] = p.col_w[cols + c * PB + k * 32];
                    if (p.col_g) gn[k] = p.col_g[cols + c * PB + k * 32];
                }
                rn = refs[c];
            };
            load_cols(0);
            for (int c = 0; c < b.nslots; c++, seq++) {
                const float u = fast_exp2(fminf(static_cast<float>(rn + bnd), MAX_EXP2));
                const float w[2] = {wn[0] * u, wn[1] * u};
                const float wg[2] = {w[0] * gn[0], w[1] * gn[1]};
                if (c + 1 < b.nslots) load_cols(c + 1);
                const int s = seq % C::NSLOT;
                if (!mbar_wait_warp<SLEEP_NS_ST>(&bar_full[s], (seq / C::NSLOT) & 1, abort_flag, WAIT_LIMIT_ST)) return false;
                uint8_t* base = smem + s * C::SLOT;
#pragma unroll
                for (int k = 0; k < 2; k++) {
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        uint4* at = reinterpret_cast<uint4*>(base + (h ? off1 : off0) + k * 32 * 128);   // (row + 32: the same row & 7)
                        uint4 raw = *at, raw2;
                        uint32_t* e = reinterpret_cast<uint32_t*>(&raw);
                        [[maybe_unused]] uint32_t* e2 = reinterpret_cast<uint32_t*>(&raw2);
#pragma unroll
                        for (int j = 0; j < 4; j++) {
                            const float2 xv = unpack2(e[j]);
                            z[h * 8 + 2 * j] = fmaf(wg[k], xv.x, z[h * 8 + 2 * j]);
                            z[h * 8 + 2 * j + 1] = fmaf(wg[k], xv.y, z[h * 8 + 2 * j + 1]);
                            const float y0 = w[k] * xv.x, y1 = w[k] * xv.y;
                            e[j] = pack2(y0, y1);
                            if constexpr (CARRY) {
                                const float2 h2 = unpack2(e[j]);
                                e2[j] = pack2(y0 - h2.x, y1 - h2.y);
                            }
                        }
                        *at = raw;
                        if constexpr (CARRY) at[C::X_BYTES / 16] = raw2;
                    }
                }
                fence_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(&bar_scaled[s]);
            }
            // the vector part: every step halves the columns a lane holds
#pragma unroll
            for (int o = 16, m = 8; m >= 1; o >>= 1, m >>= 1) {
                const bool up = (lane & o) != 0;
#pragma unroll
                for (int j = 0; j < m; j++) {
                    const float keep = up ? z[j + m] : z[j], send = up ? z[j] : z[j + m];
                    z[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                }
            }
            z[0] += __shfl_xor_sync(0xffffffffu, z[0], 1);
            if (CARRY) {
                const float d = block_decay(b0, b1);
                zrun = (d == 0.0f ? 0.0f : d * zrun) + z[0];
            } else if ((lane & 1) == 0) {
                p.vec[out] = z[0];
            }
            return true;
        });
    }
    __syncthreads();
    if (*abort_flag) {
        if (threadIdx.x == 0) atomicExch(p.status, 7000 + p.reverse);
        for (int k = 0; k < 64; k++) __nanosleep(16000);
        __syncthreads();
    }
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 2 * D);
    }
}

template <int D, int ABFMT, bool CARRY>
int launch_states_one(const BlockStateArgs& p, int dtype, cudaStream_t st) {
    using C = StCfg<D, CARRY>;
    CUtensorMap mx, my, mu;
    int rc;
    if ((rc = tc_make_map_groups(&mx, p.X, p.BH, p.S, D, dtype, false, PB, 2)) != MLSTM_OK) return rc;
    if ((rc = tc_make_map_groups(&my, p.Y, p.BH, p.S, D, dtype, false, PB, D / 64)) != MLSTM_OK) return rc;
    if ((rc = tc_make_map_out(&mu, p.U, p.BH * p.NB * C::XPARTS, D, D, dtype, 32)) != MLSTM_OK) return rc;
    auto kern = states_kernel<D, ABFMT, CARRY>;
    {   // the shared-memory opt-in is a per-device property of the kernel: set once per device
        static std::atomic<bool> opted[64];
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return MLSTM_E_CUDA;
        if (!opted[dev].load(std::memory_order_acquire)) {
            cudaError_t ce = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
            if (ce != cudaSuccess) {
                cudaGetLastError();
                return note_cuda_error(ce, "cudaFuncSetAttribute(MaxDynamicSharedMemorySize)");
            }
            opted[dev].store(true, std::memory_order_release);
        }
    }
    const long long total = static_cast<long long>(CARRY ? 1 : p.NB) * (D / TILE) * p.BH;
    if (total > 0x3fffffffLL) return MLSTM_E_SHAPE;
    const int sms = tc_sm_count();
    if (sms <= 0) return MLSTM_E_CUDA;
    const unsigned grid = static_cast<unsigned>(total < sms ? total : sms);
    cudaError_t ce = launch_pdl(kern, dim3(grid), dim3(NTHREADS_ST), C::SMEM, st, mx, my, mu, p);
    if (ce != cudaSuccess) cudaGetLastError();
    return ce == cudaSuccess ? MLSTM_OK : note_cuda_error(ce, "launch of states_kernel");
}

template <bool CARRY>
int launch_states(const BlockStateArgs& p, int D, int dtype, cudaStream_t st) {
    if (!p.U || !p.vec || p.NB <= 0 || (dtype != MLSTM_DT_BF16 && dtype != MLSTM_DT_F16)) return MLSTM_E_ARG;
    if (D != 128 && D != 256) return MLSTM_E_UNSUPPORTED;
    if (dtype == MLSTM_DT_BF16)
        return D == 128 ? launch_states_one<128, 1, CARRY>(p, dtype, st) : launch_states_one<256, 1, CARRY>(p, dtype, st);
    if constexpr (CARRY) return MLSTM_E_UNSUPPORTED;      // (a carried sum may leave fp16's range)
    else return D == 128 ? launch_states_one<128, 0, CARRY>(p, dtype, st) : launch_states_one<256, 0, CARRY>(p, dtype, st);
}

}  // namespace

int launch_block_states(const BlockStateArgs& p, int D, int dtype, cudaStream_t st) { return launch_states<false>(p, D, dtype, st); }
int launch_carried_states(const BlockStateArgs& p, int D, int dtype, cudaStream_t st) { return launch_states<true>(p, D, dtype, st); }

}  // namespace mlstm
