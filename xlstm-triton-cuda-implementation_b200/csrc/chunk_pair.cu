// Passes of the chunkwise form on CTA PAIRS (16-bit inputs, head dimension 128 or 256, blocks of an even number of
// tiles): the forward output pass (FWDC) and the three backward passes (DQC, DKC, DVC); see mlstm_common.cuh for the
// algebra and mm_tc_pair.cu for the pair protocol.  Contractions of mlstm_scan.py:200-278 (output from the carried state
// and the block's own positions) and of mlstm_matmul.py:200-316 restricted to a block.
//
// A work item is two neighbouring tiles (256 rows, one per CTA) of one block:
//   T(t) = X Y(t)^T, W = gate(T), ACC += W Z(t)     for the tiles of the block on the causal side
//   X S                                             the carried state, straight from shared memory
// and the carried part is scaled per row in fp32 (scaling X in front of the contraction would round it to 16 bits): at
// D = 128 it has an accumulator of its own and is added in the epilogue, at D = 256, where ACC fills TMEM, ACC starts
// as X S and the gate warps scale it in place.  S is read as the passes need it, from one copy in memory: FWDC and DVC
// contract over its rows (MN-major operand), DQC and DKC over its columns (K-major operand).
//
// What bounds it: HBM, as long as an item's serial chain (load, first contraction, gate, second contraction, epilogue;
// two steps per item) is covered.  Per 256 rows the tensor pipe works 6100 cycles at D = 256 (2600 at D = 128), HBM
// about 33000 (15000).  The chain runs through the gate warps, so everything is arranged around them:
//   * a pair shares every streamed tile and the state: 32 KB (16 KB) slots, and the producers run ahead into the next items;
//   * both first contractions of an item are issued before anything that needs the accumulator, i.e. under the epilogue
//     of the item before (stationary tile double at D = 128);
//   * what an item needs from the gate vectors is fetched an item ahead (loaded when the item starts: 4000 of 12500 cycles);
//   * results leave through staging and TMA stores; plain stores of the 64 KB tile held the warps for 3000 cycles;
//   * the exponential per element (16 per cycle and SM) is kept to the 32 x 32 patches of the diagonal tile that need it;
//   * items cost the same, so they are dealt out statically: no counter, no work-item messages inside the pair.
#include <atomic>
#include <type_traits>

#include "mlstm_common.cuh"
#include "ptx_sm100.cuh"
#include "tc_host.cuh"

namespace mlstm {
namespace {

using namespace ptx;

constexpr int NGROUPS = 4;
constexpr int NGATE = NGROUPS * 128;
constexpr int NTHREADS = 128 + NGATE;           // a warpgroup with the producer and the MMA warp (two warps of it idle), four gate groups
// 20 warps = five per SM sub-partition: 96 registers per thread at launch.  The gate warps' epilogue needs more (spilled
// values come back through L2, the shared memory leaves L1 nothing to speak of: 300 cycles each), so the first
// warpgroup gives most of its share away: 128 x 40 + 512 x 104 of the 640 x 96 the block is launched with.
constexpr int REGS_ROLE = 40, REGS_GATE = 104;
// An increase that the block was not launched with waits for ever, in front of every bounded wait: what the built kernel
// really has is checked on the host before its first launch.
constexpr bool register_split_fits(int regs_at_launch) {
    return REGS_ROLE <= regs_at_launch && 128 * REGS_ROLE + NGATE * REGS_GATE <= NTHREADS * regs_at_launch;
}
static_assert(register_split_fits(96), "setmaxnreg draws on the registers of the launch");
constexpr int BOX_BYTES = 128 * 128;           // 128 rows x 128 bytes
constexpr int HBOX_BYTES = 64 * 128;           // 64 rows x 128 bytes (half of a streamed Y tile's rows)
constexpr long long WAIT_LIMIT = 4000000000LL;
constexpr float MAX_ROW_EXP2 = 60.0f;          // clamp of the per-row exponent off the diagonal tile (see its use)
constexpr int SLACK_SLEEP_NS = 32;             // poll interval of the roles that wait with slack (gate warps, producer)

template <int D>
struct CpCfg {
    static constexpr bool SEP = D == 128;                       // the carried part has its own accumulator
    static constexpr int NX = D == 128 ? 2 : 1;                 // stationary-tile buffers
    static constexpr int X_BYTES = (D / 64) * BOX_BYTES;        // one stationary tile
    static constexpr int SLOT_BYTES = 128 * D;                  // Y half: 64 rows x D; Z half: 128 rows x D/2; state unit: 128 x D/2
    static constexpr int NSLOT = D == 128 ? 5 : 4;
    static constexpr int NST = D / 128;                         // slots (units of 128 contraction indices) of a state
    static constexpr int STAGE_ROW = D == 128 ? 128 : 64;       // per gate warp: 32 staging rows of that many bytes
    static constexpr int STAGE_BYTES = 32 * STAGE_ROW;
    static constexpr int OUT_BYTES = (NGATE / 32) * STAGE_BYTES;
    // per gate warp: column vectors of two steps, [2][gate, additive][32], and FWDC's vector state (D = 256 has no room for
    // them: there the lanes' values are passed round with shuffles)
    static constexpr int CVEC_FLOATS = D == 128 ? 128 + D / NGROUPS : 0;
    static constexpr int CVEC_BYTES = (NGATE / 32) * CVEC_FLOATS * 4;
    static constexpr int NPART = D == 128 ? 2 : 1;              // buffers of the row partials
    static constexpr int NBAR = 2 * NX + 2 * NSLOT + 2 + 2 + 5;
    static constexpr int HEAD_BYTES = round_up(NBAR * 8 + 64, 16);   // barriers and control words; float4 accesses follow
    static constexpr int SMEM_BYTES =
        NX * X_BYTES + NSLOT * SLOT_BYTES + OUT_BYTES + HEAD_BYTES + NPART * NGROUPS * 128 * 4 + CVEC_BYTES;
    static_assert(SMEM_BYTES <= 232448, "exceeds the shared memory of a CTA");
};

template <int MODE, int D, int ABFMT, typename OutT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(NTHREADS, 1)
mlstm_chunk_pair(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmYh,
                 const __grid_constant__ CUtensorMap tmZ, const __grid_constant__ CUtensorMap tmS,
                 const __grid_constant__ CUtensorMap tmO, const PassParams p) {
    using C = CpCfg<D>;
    using InT = typename std::conditional<ABFMT == 1, __nv_bfloat16, __half>::type;
    constexpr bool ROWS_ARE_Q = (MODE == FWDC || MODE == DQC);
    constexpr bool IS_FWD = (MODE == FWDC);
    constexpr bool IS_DQ = (MODE == DQC), IS_DK = (MODE == DKC);
    constexpr bool STATE_MN = (MODE == FWDC || MODE == DVC);    // the state step contracts over the state's rows
    static_assert(MODE == FWDC || MODE == DQC || MODE == DKC || MODE == DVC, "chunkwise passes");

    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = smem_raw;
    uint8_t* sX = smem;
    uint8_t* sSlot = sX + C::NX * C::X_BYTES;
    uint8_t* sOut = sSlot + C::NSLOT * C::SLOT_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(sOut + C::OUT_BYTES);
    uint64_t* bar_x = bars;                          // leader [NX]: both stationary tiles loaded
    uint64_t* bar_xfree = bar_x + C::NX;             // both [NX]: stationary tiles no longer read
    uint64_t* bar_full = bar_xfree + C::NX;          // leader [NSLOT]: both halves of a slot loaded
    uint64_t* bar_empty = bar_full + C::NSLOT;       // both [NSLOT]: slot no longer read by MMAs
    uint64_t* bar_t = bar_empty + C::NSLOT;          // both [2]: T tile written
    uint64_t* bar_w = bar_t + 2;                     // leader [2]: W tiles of both CTAs written (32 warp arrivals)
    uint64_t* bar_st = bar_w + 2;                    // both: X S complete (not SEP)
    uint64_t* bar_rs = bar_st + 1;                   // leader: X S scaled in both CTAs (32 warp arrivals; not SEP)
    uint64_t* bar_acc = bar_rs + 1;                  // both: accumulators complete
    uint64_t* bar_part = bar_acc + 1;                // own: row partials exchanged
    uint64_t* bar_accfree = bar_part + 1;            // leader: accumulators of both CTAs drained (32 warp arrivals)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + C::NBAR);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    float* part_base = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(bars) + C::HEAD_BYTES);  // [NPART][NGROUPS][128]
    float* cvec_base = part_base + C::NPART * NGROUPS * 128;

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();    // 0 = leader
    const uint32_t peer = rank ^ 1u;
    const int NT = p.Spad / TILE;
    const int NP = (NT + 1) / 2;                 // tile pairs per slice
    const int total = NP * p.BH;
    const int npairs = gridDim.x >> 1;
    const int nparts = p.state_parts == 2 ? 2 : 1;   // 16-bit halves of the carried state
    const bool misaligned = (smem_u32(smem) & 1023u) != 0;   // uniform over the cluster in practice; never seen

    struct Item {
        int bh, pair, tile, blk, first, nsteps;
    };
    auto decode = [&](int id) {
        Item it;
        it.bh = id / NP;
        it.pair = id - it.bh * NP;
        it.tile = 2 * it.pair + static_cast<int>(rank);     // this CTA's stationary tile (may be == NT: idle half)
        it.blk = (2 * it.pair) / p.chunk_tiles;             // chunk_tiles is even: both tiles are of one block
        it.first = it.blk * p.chunk_tiles;
        const int end = min(it.first + p.chunk_tiles, NT);
        it.nsteps = ROWS_ARE_Q ? min(2 * it.pair + 2, NT) - it.first : end - 2 * it.pair;
        return it;
    };
    auto stream_tile = [&](const Item& it, int t) { return ROWS_ARE_Q ? it.first + t : 2 * it.pair + t; };
    // shared::cluster addresses of the leader's and the peer's copies of a barrier
    auto at_leader = [&](const void* local) { return mapa_u32(smem_u32(local), 0u); };
    auto at_peer = [&](const void* local) { return mapa_u32(smem_u32(local), peer); };

    if (threadIdx.x == 0) {
        for (int s = 0; s < C::NX; s++) {
            mbar_init(&bar_x[s], 1);
            mbar_init(&bar_xfree[s], IS_FWD ? 1 + NGATE / 32 : 1);   // FWDC: the gate warps read the query tile as well
        }
        for (int s = 0; s < C::NSLOT; s++) {
            mbar_init(&bar_full[s], 1);
            mbar_init(&bar_empty[s], 1);
        }
        for (int s = 0; s < 2; s++) {
            mbar_init(&bar_t[s], 1);
            mbar_init(&bar_w[s], 2 * NGATE / 32);
        }
        mbar_init(bar_st, 1);
        mbar_init(bar_acc, 1);
        mbar_init(bar_part, NGATE / 32);
        mbar_init(bar_rs, 2 * NGATE / 32);
        mbar_init(bar_accfree, 2 * NGATE / 32);
        *abort_flag = misaligned ? 1 : 0;
        fence_mbar_init();
    }
    if (warp == 1) {
        tmem_alloc_pair(tmem_slot, 512);
        tmem_relinquish_pair();
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();           // the peer's barriers are initialised before anything signals them
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tmem_T0 = tmem_base;
    const uint32_t tmem_ACC = tmem_base + 256;
    const uint32_t tmem_CAR = tmem_ACC + (C::SEP ? D : 0);    // X S
    // nothing above touched global memory (see grid_dep_wait in mlstm_common.cuh)
    grid_dep_wait();
    grid_dep_launch();

    if (warp < 4) {
    set_max_regs_dec<REGS_ROLE>();
    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer (one per CTA)
        if (lane == 0) {
            prefetch_tmap(&tmX);
            prefetch_tmap(&tmYh);
            prefetch_tmap(&tmZ);
            prefetch_tmap(&tmS);
            int slot_it = 0;
            bool ok = !*abort_flag;
            // the next slot, free to be written, with the bytes of both CTAs announced on the leader's barrier
            auto open_slot = [&](uint8_t*& dst, uint32_t& lead_full) {
                const int s = slot_it % C::NSLOT;
                ok = ok && mbar_wait<SLACK_SLEEP_NS>(&bar_empty[s], ((slot_it / C::NSLOT) & 1) ^ 1, abort_flag, WAIT_LIMIT);
                if (!ok) return false;
                if (rank == 0) mbar_expect_tx(&bar_full[s], 2 * C::SLOT_BYTES);
                lead_full = at_leader(&bar_full[s]);
                dst = sSlot + s * C::SLOT_BYTES;
                slot_it++;
                return true;
            };
            int n = 0;
            for (int id = blockIdx.x >> 1; id < total && ok; id += npairs, n++) {
                const Item it = decode(id);
                const int xb = n % C::NX;
                ok = mbar_wait<SLACK_SLEEP_NS>(&bar_xfree[xb], ((n / C::NX) & 1) ^ 1, abort_flag, WAIT_LIMIT);
                if (!ok) break;
                if (rank == 0) mbar_expect_tx(&bar_x[xb], 2 * C::X_BYTES);
                const uint32_t lead_x = at_leader(&bar_x[xb]);
                for (int c = 0; c < D / 64; c++)   // rows past the end of the slice (idle half, ragged S) read as zeros
                    tma_load_3d_pair(sX + xb * C::X_BYTES + c * BOX_BYTES, &tmX, lead_x, c * 64, it.tile * TILE, it.bh);
                uint8_t* dst;
                uint32_t lead_full;
                auto load_y = [&](int t) {   // this CTA's 64 rows of the streamed tile, all columns
                    if (!open_slot(dst, lead_full)) return;
                    const int row = stream_tile(it, t) * TILE + static_cast<int>(rank) * 64;
                    for (int c = 0; c < D / 64; c++) tma_load_3d_pair(dst + c * HBOX_BYTES, &tmYh, lead_full, c * 64, row, it.bh);
                };
                auto load_z = [&](int t) {   // all 128 rows of the streamed tile, this CTA's half of the columns
                    if (!open_slot(dst, lead_full)) return;
                    for (int c = 0; c < D / 128; c++)
                        tma_load_3d_pair(dst + c * BOX_BYTES, &tmZ, lead_full, static_cast<int>(rank) * (D / 2) + c * 64,
                                         stream_tile(it, t) * TILE, it.bh);
                };
                auto load_state = [&](int part, int u) {   // contraction indices [128 u, 128 u + 128), this CTA's half of the outputs
                    if (!open_slot(dst, lead_full)) return;
                    const int z = (it.bh * p.NB + it.blk) * nparts + part;
                    if (STATE_MN) {
                        for (int c = 0; c < D / 128; c++)
                            tma_load_3d_pair(dst + c * BOX_BYTES, &tmS, lead_full, static_cast<int>(rank) * (D / 2) + c * 64, u * 128, z);
                    } else {
                        for (int c = 0; c < 2; c++)
                            tma_load_3d_pair(dst + c * (D / 2 * 128), &tmS, lead_full, u * 128 + c * 64, static_cast<int>(rank) * (D / 2), z);
                    }
                };
                // same order as the MMA issuer consumes
                load_y(0);
                if (it.nsteps > 1) load_y(1);
                for (int part = 0; part < nparts; part++)
                    for (int u = 0; u < C::NST; u++) load_state(part, u);
                for (int t = 2; t < it.nsteps && ok; t++) {
                    load_z(t - 2);
                    load_y(t);
                }
                if (it.nsteps > 1) load_z(it.nsteps - 2);
                load_z(it.nsteps - 1);
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer (leader only)
        // the whole warp runs the loop, one elected lane issues (see mm_tc.cu for why)
        if (rank == 0) {
            const bool issuer = elect_one();
            auto uni = [](int x) { return __shfl_sync(0xffffffffu, x, 0); };
            auto wait_u = [&](uint64_t* bar, uint32_t parity) { return mbar_wait_warp(bar, parity, abort_flag, WAIT_LIMIT); };
            constexpr uint32_t idesc_t = make_idesc(ABFMT, 256, 128, 0, 0);
            constexpr uint32_t idesc_z = make_idesc(ABFMT, 256, D, 0, 1);
            constexpr uint32_t idesc_s = make_idesc(ABFMT, 256, D, 0, STATE_MN ? 1 : 0);
            const uint32_t sX_u = static_cast<uint32_t>(uni(static_cast<int>(smem_u32(sX))));
            const uint32_t sSlot_u = sX_u + C::NX * C::X_BYTES;
            const uint32_t bars_u = sSlot_u + C::NSLOT * C::SLOT_BYTES + C::OUT_BYTES;   // this CTA's barriers ...
            const uint32_t bars_peer_u = static_cast<uint32_t>(uni(static_cast<int>(at_peer(bars))));   // ... and the peer's
            const uint32_t tmem_T0u = static_cast<uint32_t>(uni(static_cast<int>(tmem_T0)));
            const uint64_t xdesc0 = smem_desc_sw128(sX_u, 16, 1024);
            const uint64_t kdesc0 = smem_desc_sw128(sSlot_u, 16, 1024);               // K-major view of slot 0
            const uint64_t mndesc0 = smem_desc_sw128(sSlot_u, BOX_BYTES, 1024, 2);    // MN-major view of slot 0
            auto commit_both = [&](const uint64_t* bar) {   // one arrival in either CTA
                const uint32_t off = static_cast<uint32_t>(bar - bars) * 8u;
                tc_commit_pair(bars_u + off);
                tc_commit_pair(bars_peer_u + off);
            };
            int slot_it = 0;
            int gstep = 0;
            int n = 0;
            bool ok = __all_sync(0xffffffffu, *abort_flag ? 0 : 1) != 0;
            for (int id = blockIdx.x >> 1; id < total && ok; id += npairs, n++) {
                const Item it = decode(id);
                const int xb = n % C::NX;
                const uint32_t acc = tmem_T0u + 256, car = acc + (C::SEP ? D : 0);
                const uint64_t xdesc = smem_desc_advance(xdesc0, xb * C::X_BYTES);
                ok = wait_u(&bar_x[xb], (n / C::NX) & 1);
                if (!ok) break;
                tc_fence_after();
                auto first = [&](int t) {   // T(t) = X Y(t)^T: N = 128 (64 rows of Y from each CTA)
                    const int gt = gstep + t;
                    const uint32_t t_tmem = tmem_T0u + (gt & 1) * 128;
                    const int s = slot_it % C::NSLOT;
                    ok = ok && wait_u(&bar_full[s], (slot_it / C::NSLOT) & 1);
                    if (!ok) return;
                    const uint64_t yd = smem_desc_advance(kdesc0, s * C::SLOT_BYTES);
                    if (issuer) {
#pragma unroll
                        for (int kx = 0; kx < D / 16; kx++)
                            mma_ss_pair(t_tmem, smem_desc_advance(xdesc, (kx >> 2) * BOX_BYTES + (kx & 3) * 32),
                                        smem_desc_advance(yd, (kx >> 2) * HBOX_BYTES + (kx & 3) * 32), idesc_t, kx > 0 ? 1u : 0u);
                        commit_both(&bar_t[gt & 1]);
                        commit_both(&bar_empty[s]);
                        if (t == it.nsteps - 1 && t > 1) commit_both(&bar_xfree[xb]);   // (up to two steps: after X S)
                    }
                    __syncwarp();
                    slot_it++;
                };
                auto state = [&]() {   // X S
                    ok = ok && wait_u(bar_accfree, (n & 1) ^ 1);
                    if (!ok) return;
                    tc_fence_after();
#pragma unroll 1
                    for (int part = 0; part < nparts; part++) {
#pragma unroll
                        for (int u = 0; u < C::NST; u++) {
                            const int s = slot_it % C::NSLOT;
                            ok = wait_u(&bar_full[s], (slot_it / C::NSLOT) & 1);
                            if (!ok) return;
                            const uint64_t sd = smem_desc_advance(STATE_MN ? mndesc0 : kdesc0, s * C::SLOT_BYTES);
                            if (issuer) {
#pragma unroll
                                for (int kk = 0; kk < 8; kk++) {
                                    const int kx = u * 8 + kk;
                                    mma_ss_pair(car, smem_desc_advance(xdesc, (kx >> 2) * BOX_BYTES + (kx & 3) * 32),
                                                smem_desc_advance(sd, STATE_MN ? kk * 2048 : (kk >> 2) * (D / 2 * 128) + (kk & 3) * 32),
                                                idesc_s, (part > 0 || kx > 0) ? 1u : 0u);
                                }
                                if (part == nparts - 1 && u == C::NST - 1) {
                                    if (!C::SEP) commit_both(bar_st);
                                    if (it.nsteps <= 2) commit_both(&bar_xfree[xb]);
                                }
                                commit_both(&bar_empty[s]);
                            }
                            __syncwarp();
                            slot_it++;
                        }
                    }
                };
                auto second = [&](int u) {  // ACC += W(u) Z(u), both CTAs
                    const int gu = gstep + u;
                    ok = ok && wait_u(&bar_w[gu & 1], (gu >> 1) & 1);
                    if (!ok) return;
                    tc_fence_after();
                    const int s = slot_it % C::NSLOT;
                    ok = wait_u(&bar_full[s], (slot_it / C::NSLOT) & 1);
                    if (!ok) return;
                    if (!C::SEP && u == 0) {
                        ok = wait_u(bar_rs, n & 1);
                        if (!ok) return;
                        tc_fence_after();
                    }
                    const uint32_t w_tmem = tmem_T0u + (gu & 1) * 128;
                    const uint64_t zd = smem_desc_advance(mndesc0, s * C::SLOT_BYTES);
                    if (issuer) {
#pragma unroll
                        for (int kk = 0; kk < 8; kk++)   // 16 streamed rows per MMA
                            mma_ts_pair(acc, w_tmem + (kk >> 1) * 32 + (kk & 1) * 8, smem_desc_advance(zd, kk * 2048), idesc_z,
                                        (!C::SEP || u > 0 || kk > 0) ? 1u : 0u);
                        if (u == it.nsteps - 1) commit_both(bar_acc);
                        commit_both(&bar_empty[s]);
                    }
                    __syncwarp();
                    slot_it++;
                };
                first(0);
                if (it.nsteps > 1) first(1);
                state();
                for (int t = 2; t < it.nsteps && ok; t++) {
                    second(t - 2);
                    first(t);
                }
                if (it.nsteps > 1) second(it.nsteps - 2);
                second(it.nsteps - 1);
                gstep += it.nsteps;
            }
        }
    }
    } else {
        // ------------------------------------------------------------ gate groups
        set_max_regs_inc<REGS_GATE>();
        const int grp = (warp - 4) >> 2;
        const int q32 = (warp & 3) * 32;               // this warp's rows inside the tile
        const int r = q32 + lane;                      // TMEM lane == row inside the tile
        const uint32_t lane_bits = static_cast<uint32_t>(q32) << 16;
        const int cbase = grp * 32;                    // this group's columns of a T tile
        constexpr int QUART = D / NGROUPS;             // this group's columns of the accumulator
        constexpr int NCH = QUART / 32;
        const int c0 = grp * QUART;
        const uint32_t lead_w[2] = {at_leader(&bar_w[0]), at_leader(&bar_w[1])};
        const uint32_t lead_accfree = at_leader(bar_accfree);
        bool ok = __all_sync(0xffffffffu, *abort_flag == 0) != 0;
        int gstep = 0;
        uint8_t* stage = sOut + (warp - 4) * C::STAGE_BYTES;                  // rows on their way out (or in: q, k, o)
        [[maybe_unused]] float* cvec = cvec_base + (warp - 4) * C::CVEC_FLOATS;
        [[maybe_unused]] float* zvec = cvec + 128;
        if (lane == 0) prefetch_tmap(&tmO);
        // entry j of a vector whose lane values are `own` (and, where there is room, lie in shared memory at `vec`)
        auto four = [&](const float* vec, float own, int j4, float (&out)[4]) {
            if constexpr (C::CVEC_FLOATS > 0) {
                const float4 v = *reinterpret_cast<const float4*>(vec + j4 * 4);
                out[0] = v.x; out[1] = v.y; out[2] = v.z; out[3] = v.w;
            } else {
#pragma unroll
                for (int k = 0; k < 4; k++) out[k] = __shfl_sync(0xffffffffu, own, j4 * 4 + k);
            }
        };

        // Everything an item needs from the gate vectors is requested one item ahead, after the last gate step of the item
        // before (load), and reduced to a few floats at its accumulator wait (combine): a warp that loads them when the item
        // starts waits for L2 again and again, 4000 of 12500 cycles per item.
        struct Raw {
            float rel;
            double ref, b, lb, cr[2];
        };
        struct Terms {
            float er[2];         // row part of the exponent for steps 0 and 1
            float state_w;       // row weight of the carried state
            float m;             // FWDC: the row's stabiliser
            float g;             // DQC: additive term
            float w[2], gc[2];   // lane j: gate term (and DKC's additive term) of column cbase + j in steps 0 and 1
            float z[NCH];        // lane j: vector state at column c0 + 32 ch + j
        };
        // Lane j's column of step t, as a factor, except where the patch needs the exponent itself: on the diagonal tile, if its
        // columns' 64-position reference block is also the rows' (a masked column can then lie above the row's maximum).
        const bool diag_exact = (grp >> 1) == ((warp & 3) >> 1);
        auto column_term = [&](const Item& it, int t) {
            const int st = stream_tile(it, t);
            return (st == it.tile && diag_exact ? p.col_rel : p.col_w)[static_cast<size_t>(it.bh) * p.Spad + st * TILE + cbase + lane];
        };
        auto column_ref = [&](const Item& it, int t) {
            return p.col_ref[static_cast<size_t>(it.bh) * (p.Spad / REF_BLOCK) + stream_tile(it, t) * (TILE / REF_BLOCK) + (grp >> 1)];
        };
        auto load_terms = [&](const Item& it, Raw& rr, Terms& tm) {
            const size_t vec_base = static_cast<size_t>(it.bh) * p.Spad;
            const int grow = min(it.tile, NT - 1) * TILE + r;      // (the idle half reads its partner's rows and uses nothing)
            rr.rel = p.row_rel[vec_base + grow];
            rr.ref = p.row_ref[static_cast<size_t>(it.bh) * (p.Spad / REF_BLOCK) + grow / REF_BLOCK];
            rr.b = p.An_bound[static_cast<size_t>(it.bh) * (p.NB + 1) + it.blk + (ROWS_ARE_Q ? 0 : 1)];
            // (no branch around a load: merging its two outcomes would wait for it here)
            if (IS_FWD) rr.lb = *(p.late_bound ? p.late_bound + it.bh : p.An_bound);
            const int t1 = min(1, it.nsteps - 1);
            rr.cr[0] = column_ref(it, 0);
            rr.cr[1] = column_ref(it, t1);
            tm.w[0] = column_term(it, 0);
            tm.w[1] = column_term(it, t1);
            if (IS_DK) {
                tm.gc[0] = p.col_g[vec_base + stream_tile(it, 0) * TILE + cbase + lane];
                tm.gc[1] = p.col_g[vec_base + stream_tile(it, t1) * TILE + cbase + lane];
            }
            if (IS_FWD) tm.m = p.m[static_cast<size_t>(it.bh) * p.S + min(grow, p.S - 1)];
            if (IS_DQ) tm.g = p.row_g[vec_base + grow];
            if (MODE != DVC) {
                const float* zv = (IS_DK ? p.rvec : p.zstate) + (static_cast<size_t>(it.bh) * p.NB + it.blk) * D + c0 + lane;
#pragma unroll
                for (int ch = 0; ch < NCH; ch++) tm.z[ch] = zv[ch * 32];
            }
        };
        // FWDC with a late carry: the row's stabiliser and the inbound boundary are capped by the carried-in maximum, and m
        // grows by what the cap took off.  A row without a finite gate of its own (rel = -inf: left padding, gates.cu) has the
        // carried-in maximum, if there is one, and then an m that is not known here (NaN: it takes no part in the normaliser).
        auto capped = [&](float rel, double negA, double lb) {
            return rel == -INFINITY && lb < static_cast<double>(INFINITY) ? lb : fmin(negA, lb);
        };
        // Row weight of the carried state: FWDC, DQC exp(A_end(k-1) - A_t) (times scale, resp. scale / n_t); DKC, DVC
        // exp(a_j - A_end(k)); 0 where nothing is carried in, and for a position whose weights are all 0.
        auto combine = [&](const Item& it, const Raw& rr, Terms& tm) {
            double negA = static_cast<double>(rr.rel) + rr.ref, bound = rr.b;
            const bool none = it.tile >= NT || (rr.rel == -INFINITY && !(IS_FWD && p.late_bound));
            if (IS_FWD && p.late_bound) {
                const double negA_c = capped(rr.rel, negA, rr.lb);
                tm.m = negA < negA_c ? NAN : tm.m + static_cast<float>((negA - negA_c) * 0.6931471805599453);
                negA = negA_c;
                bound = fmin(bound, rr.lb);
            }
            const double er_d = negA + static_cast<double>(p.er_add);
            tm.er[0] = static_cast<float>(er_d + rr.cr[0]);
            tm.er[1] = static_cast<float>(er_d + rr.cr[1]);
            tm.state_w = none ? 0.0f : fast_exp2(static_cast<float>(ROWS_ARE_Q ? er_d - bound : er_d + bound));
        };
        // (plain loads, no __ldg: the first item's are not to move in front of grid_dep_wait)
        Raw raw{};
        Terms nx{};
        Item it = decode(blockIdx.x >> 1);
        load_terms(it, raw, nx);
        combine(it, raw, nx);

        int n = 0;
        for (int id = blockIdx.x >> 1; id < total && ok; id += npairs, n++) {
            const Terms tm = nx;
            const int bh = it.bh, tile = it.tile, nsteps = it.nsteps;
            const bool active = tile < NT;             // the idle half of an odd last pair only keeps the protocol going
            float rowsum = 0.0f;
            if constexpr (C::CVEC_FLOATS > 0) {
                __syncwarp();
#pragma unroll
                for (int t = 0; t < 2; t++) {
                    cvec[t * 64 + lane] = tm.w[t];
                    if (IS_DK) cvec[t * 64 + 32 + lane] = tm.gc[t];
                }
                if (MODE != DVC) zvec[lane] = tm.z[0];
                __syncwarp();
            } else if constexpr (IS_DQ || IS_DK) {
                // The vector of the epilogue's rank-1 term, where FWDC has its row partials: every warp of a group writes the same
                // values and reads its own.  Two buffers: a warp two items ahead has seen every warp of the pair scale the item
                // between (bar_rs), i.e. leave this one.
                zvec = part_base + (n & 1) * (NGROUPS * QUART) + c0;
                __syncwarp();
#pragma unroll
                for (int ch = 0; ch < NCH; ch++) zvec[ch * 32 + lane] = tm.z[ch];
                __syncwarp();
            }

            // the carried part, X S: its share of the normaliser (FWDC) and, where it sits in ACC, its row weight
            auto carried = [&]() {
                if constexpr (IS_FWD) {
                    // w (q . z) over this group's columns: q from the stationary tile (128-byte swizzle: 16-byte piece j of row
                    // r sits at piece j ^ (r & 7))
                    const uint8_t* xrow = sX + (n % C::NX) * C::X_BYTES + (c0 / 64) * BOX_BYTES + r * 128;
                    float qz = 0.0f;
#pragma unroll
                    for (int j8 = 0; j8 < QUART / 8; j8++) {
                        const int piece = (c0 % 64) / 8 + j8;
                        const uint4 raw16 = *reinterpret_cast<const uint4*>(xrow + ((piece ^ (r & 7)) << 4));
                        const InT* qv = reinterpret_cast<const InT*>(&raw16);
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            float z4[4];
                            four(zvec, tm.z[j8 / 4], (j8 % 4) * 2 + h, z4);
#pragma unroll
                            for (int k = 0; k < 4; k++) qz = fmaf(to_f32<InT>(qv[h * 4 + k]), z4[k], qz);
                        }
                    }
                    if (tm.state_w != 0.0f) rowsum = fmaf(tm.state_w, qz, rowsum);
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&bar_xfree[n % C::NX]);
                }
                if constexpr (!C::SEP) {
                    ok = mbar_wait_warp<SLACK_SLEEP_NS>(bar_st, n & 1, abort_flag, WAIT_LIMIT);
                    if (!ok) return;
                    tc_fence_after();
                    const bool none = __all_sync(0xffffffffu, tm.state_w == 0.0f);   // nothing carried in (or an idle half)
#pragma unroll 1
                    for (int ch = 0; ch < NCH; ch++) {
                        const uint32_t at = tmem_CAR + lane_bits + c0 + ch * 32;
                        uint32_t av[32];
                        tmem_ld32(at, av);
                        tc_wait_ld();
#pragma unroll
                        for (int j = 0; j < 32; j++) av[j] = none ? 0u : __float_as_uint(__uint_as_float(av[j]) * tm.state_w);
                        tmem_st32(at, av);
                    }
                    tc_wait_st();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_remote(at_leader(bar_rs));
                }
            };

            for (int t = 0; t < nsteps; t++) {
                const int gt = gstep + t;
                const int buf = gt & 1;
                const int st = stream_tile(it, t);
                const bool diag = (st == tile);
                // tiles on the wrong side of this CTA's diagonal (they belong to the partner's triangle) give W = 0, and so
                // does, on the diagonal tile, a 32 x 32 patch that lies wholly on the masked side
                const bool dead = !active || (ROWS_ARE_Q ? (st > tile) : (st < tile)) ||
                                  (diag && (ROWS_ARE_Q ? (grp > (warp & 3)) : (grp < (warp & 3))));
                const bool exact = diag && diag_exact;
                float er = t == 0 ? tm.er[0] : tm.er[1];
                float w_own = t == 0 ? tm.w[0] : tm.w[1];
                float g_own = IS_DK ? (t == 0 ? tm.gc[0] : tm.gc[1]) : 0.0f;
                [[maybe_unused]] float* cv = cvec + (t & 1) * 64;
                if (t >= 2 && !dead) {                 // blocks of more than two tiles
                    const size_t vec_base = static_cast<size_t>(bh) * p.Spad;
                    const int grow = tile * TILE + r;
                    double negA = static_cast<double>(p.row_rel[vec_base + grow]) +
                                  p.row_ref[static_cast<size_t>(bh) * (p.Spad / REF_BLOCK) + grow / REF_BLOCK];
                    if (IS_FWD && p.late_bound) negA = capped(p.row_rel[vec_base + grow], negA, p.late_bound[bh]);
                    er = static_cast<float>(negA + static_cast<double>(p.er_add) + column_ref(it, t));
                    w_own = column_term(it, t);
                    if (IS_DK) g_own = p.col_g[vec_base + st * TILE + cbase + lane];
                    if constexpr (C::CVEC_FLOATS > 0) {
                        __syncwarp();
                        cv[lane] = w_own;
                        if (IS_DK) cv[32 + lane] = g_own;
                        __syncwarp();
                    }
                }
                ok = mbar_wait_warp<SLACK_SLEEP_NS>(&bar_t[buf], (gt >> 1) & 1, abort_flag, WAIT_LIMIT);
                if (!ok) break;
                tc_fence_after();
                const uint32_t t_tmem = tmem_T0 + buf * 128 + lane_bits + cbase;
                uint32_t pk[16];
                if (dead) {
#pragma unroll
                    for (int j = 0; j < 16; j++) pk[j] = 0u;
                } else {
                    uint32_t tv[32];
                    tmem_ld32(t_tmem, tv);
                    tc_wait_ld();
                    // exp2(ec + er) = exp2(ec) exp2(er), both bounded; a 64-column block of pure padding has no reference of its
                    // own, hence the clamp (its column factors are 0)
                    const float u = fast_exp2(fminf(er, MAX_ROW_EXP2));
#pragma unroll
                    for (int j4 = 0; j4 < 8; j4++) {
                        float ce[4], ge[4], w4[4];
                        four(cv, w_own, j4, ce);
                        if (IS_DK) four(cv + 32, g_own, j4, ge);
#pragma unroll
                        for (int jj = 0; jj < 4; jj++) {
                            const int j = j4 * 4 + jj;
                            float tval = __uint_as_float(tv[j]);
                            if (IS_DQ) tval += tm.g;
                            if (IS_DK) tval += ge[jj];
                            float wj;
                            if (exact) {
                                wj = tval * fast_exp2(ce[jj] + er);
                                if (ROWS_ARE_Q ? (cbase + j > r) : (cbase + j < r)) wj = 0.0f;
                            } else {
                                wj = tval * u * ce[jj];
                            }
                            if (IS_FWD) rowsum += wj;
                            w4[jj] = wj;
                        }
#pragma unroll
                        for (int jj = 0; jj < 2; jj++) {
                            if constexpr (ABFMT == 1) {
                                __nv_bfloat162 v2 = __floats2bfloat162_rn(w4[2 * jj], w4[2 * jj + 1]);
                                pk[j4 * 2 + jj] = *reinterpret_cast<uint32_t*>(&v2);
                            } else {
                                __half2 v2 = __floats2half2_rn(w4[2 * jj], w4[2 * jj + 1]);
                                pk[j4 * 2 + jj] = *reinterpret_cast<uint32_t*>(&v2);
                            }
                        }
                    }
                }
                tmem_st16(t_tmem, pk);
                tc_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_remote(lead_w[buf]);
                if (t == 1 || nsteps == 1) {           // after the first two gates: X S is issued behind both first contractions
                    carried();
                    if (!ok) break;
                }
            }
            if (!ok) break;
            gstep += nsteps;

            // ---- while the last contractions run: everything of the epilogue that does not need the accumulator
            // Row partials: nobody still reads what this buffer held before.  D = 256: a warp is past "X S complete", which
            // follows the drain of the accumulator (and with it the reading) by every warp an item ago; D = 128: two items ago,
            // by the accumulator wait of the item before.
            [[maybe_unused]] float* part = part_base + (n % C::NPART) * NGROUPS * 128;
            if constexpr (IS_FWD) {
                part[grp * 128 + r] = rowsum;
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_part);
            }
            const Item it_next = decode(min(id + npairs, total - 1));
            load_terms(it_next, raw, nx);
            const int row0 = tile * TILE + q32;
            const int nrows = active ? min(32, p.S - row0) : 0;            // (may be negative)
            // What the rows are dotted with (DQC: q, DKC: k) or gated by (FWDC: o): 32 rows x 64 bytes per chunk, LDG of eight
            // whole row pieces per instruction, requested before the accumulator wait and turned to one row per lane in staging.
            const void* side_src = IS_FWD ? p.ogate : (IS_DQ || IS_DK) ? p.dot_src : nullptr;
            uint4 sd[4];
            auto load_side = [&](int ch) {
                const InT* src = reinterpret_cast<const InT*>(side_src) + (static_cast<size_t>(bh) * p.S + row0) * D + c0 + ch * 32;
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const int row = k * 8 + (lane >> 2);
                    sd[k] = make_uint4(0u, 0u, 0u, 0u);
                    if (row < nrows) sd[k] = ld_global_nc_v4(src + static_cast<size_t>(row) * D + (lane & 3) * 8);
                }
            };
            if (side_src) load_side(0);
            float inv_n = 1.0f;
            if constexpr (IS_FWD) {
                ok = mbar_wait_warp<SLACK_SLEEP_NS>(bar_part, n & 1, abort_flag, WAIT_LIMIT);
                if (!ok) break;
                const float bsum = (part[r] + part[128 + r]) + (part[256 + r] + part[384 + r]);
                inv_n = 1.0f / (fmaxf(fabsf(bsum), __expf(-tm.m)) + 1e-6f);
                if (grp == 0 && lane < nrows && p.b_out) p.b_out[static_cast<size_t>(bh) * p.S + row0 + lane] = bsum;
            }

            // ---- epilogue: each group drains a quarter of this CTA's accumulator columns
            ok = mbar_wait_warp<SLACK_SLEEP_NS>(bar_acc, n & 1, abort_flag, WAIT_LIMIT);
            if (!ok) break;
            tc_fence_after();
            combine(it_next, raw, nx);
            float dot = 0.0f;
            // DQC / DKC: what the carried state leaves out is a rank-1 term, coef * vec[column]:
            //   dQ_t += beta_t g_t z_k    (the db part of the carried-in state, z_k the inbound normaliser vector)
            //   dK_j += gamma_j r_k       (r_k: the same part of the state carried back from the later blocks)
            [[maybe_unused]] const float rank1_coef = IS_DQ ? tm.state_w * tm.g : tm.state_w;
            // this warp's 32 rows x 32 columns (x the first of them) to global memory through its staging rows (16-byte pieces
            // swizzled over the bank groups, as the tensor map has it); rows past the end of the slice are not written
            auto store_chunk = [&](const uint32_t (&v)[32], int x) {
                constexpr int RB = sizeof(OutT) == 4 ? C::STAGE_ROW : 64;
                constexpr int CPS = RB / static_cast<int>(sizeof(OutT));      // columns per store
#pragma unroll
                for (int sub = 0; sub < 32 / CPS; sub++) {
                    if (lane == 0) bulk_wait_read_all();   // the previous store has read the staging rows
                    __syncwarp();
                    uint8_t* srow = stage + lane * RB;
                    const int sw = RB == 128 ? (lane & 7) : ((lane >> 1) & 3);
#pragma unroll
                    for (int j = 0; j < RB / 16; j++) {
                        uint4 w;
                        if constexpr (sizeof(OutT) == 4) {
                            w = make_uint4(v[sub * CPS + j * 4], v[sub * CPS + j * 4 + 1], v[sub * CPS + j * 4 + 2], v[sub * CPS + j * 4 + 3]);
                        } else {
                            uint32_t o32[4];
#pragma unroll
                            for (int k = 0; k < 4; k++) {
                                const float lo = __uint_as_float(v[j * 8 + 2 * k]), hi = __uint_as_float(v[j * 8 + 2 * k + 1]);
                                if constexpr (ABFMT == 1) {
                                    __nv_bfloat162 v2 = __floats2bfloat162_rn(lo, hi);
                                    o32[k] = *reinterpret_cast<uint32_t*>(&v2);
                                } else {
                                    __half2 v2 = __floats2half2_rn(lo, hi);
                                    o32[k] = *reinterpret_cast<uint32_t*>(&v2);
                                }
                            }
                            w = make_uint4(o32[0], o32[1], o32[2], o32[3]);
                        }
                        *reinterpret_cast<uint4*>(srow + ((j ^ sw) << 4)) = w;
                    }
                    fence_async_smem();
                    __syncwarp();
                    if (lane == 0 && active) {
                        tma_store_3d(&tmO, stage, x + sub * CPS, row0, bh);
                        bulk_commit();
                    }
                }
            };
#pragma unroll
            for (int ch = 0; ch < NCH; ch++) {
                uint32_t av[32];
                tmem_ld32(tmem_ACC + lane_bits + c0 + ch * 32, av);
                if constexpr (C::SEP) {
#pragma unroll
                    for (int h = 0; h < 2; h++) {      // (in halves: 64 values at once do not fit the registers)
                        uint32_t sv[16];
                        tmem_ld16(tmem_CAR + lane_bits + c0 + h * 16, sv);
                        tc_wait_ld();
                        if (!__all_sync(0xffffffffu, tm.state_w == 0.0f)) {
#pragma unroll
                            for (int j = 0; j < 16; j++)
                                av[h * 16 + j] = __float_as_uint(fmaf(__uint_as_float(sv[j]), tm.state_w, __uint_as_float(av[h * 16 + j])));
                        }
                    }
                } else {
                    tc_wait_ld();
                }
                if (ch == NCH - 1) {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_remote(lead_accfree);
                }
                if constexpr (IS_FWD) {
#pragma unroll
                    for (int j = 0; j < 32; j++) av[j] = __float_as_uint(__uint_as_float(av[j]) * inv_n);
                }
                if (side_src) {
                    if (lane == 0) bulk_wait_read_all();
                    __syncwarp();
#pragma unroll
                    for (int k = 0; k < 4; k++) {   // 64-byte rows, 16-byte pieces swizzled over the bank groups
                        const int row = k * 8 + (lane >> 2);
                        *reinterpret_cast<uint4*>(stage + row * 64 + (((lane & 3) ^ ((row >> 1) & 3)) << 4)) = sd[k];
                    }
                    __syncwarp();
                    if (ch + 1 < NCH) load_side(ch + 1);
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const uint4 raw16 = *reinterpret_cast<const uint4*>(stage + lane * 64 + ((k ^ ((lane >> 1) & 3)) << 4));
                        const InT* ev = reinterpret_cast<const InT*>(&raw16);
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            float z4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                            if constexpr (!IS_FWD) {
                                const float4 v = *reinterpret_cast<const float4*>(zvec + ch * 32 + k * 8 + h * 4);
                                z4[0] = v.x; z4[1] = v.y; z4[2] = v.z; z4[3] = v.w;
                            }
#pragma unroll
                            for (int jj = 0; jj < 4; jj++) {
                                const int j = h * 4 + jj;
                                float x = __uint_as_float(av[k * 8 + j]);
                                if (IS_FWD) {
                                    x *= silu_f(to_f32<InT>(ev[j]));
                                } else {
                                    x = fmaf(rank1_coef, z4[jj], x);
                                    dot = fmaf(x, to_f32<InT>(ev[j]), dot);
                                }
                                av[k * 8 + j] = __float_as_uint(x);
                            }
                        }
                    }
                    __syncwarp();
                }
                store_chunk(av, c0 + ch * 32);
            }
            // one partial per gate group: adding them up is left to the dF kernel, so that the groups need not meet here
            if ((IS_DQ || IS_DK) && p.dot_out && active)
                p.dot_out[grp * p.dot_part_stride + static_cast<long long>(bh) * p.Spad + row0 + lane] = lane < nrows ? dot : 0.0f;
            it = it_next;
        }
        if (lane == 0) bulk_wait_all();   // the last stores have left shared memory before the CTA goes away
        tc_fence_before();
    }

    __syncthreads();
    if (*abort_flag) {
        if (threadIdx.x == 0) atomicExch(p.status, misaligned ? 2000 : 6000 + MODE);
        for (int k = 0; k < 64; k++) __nanosleep(16000);
        __syncthreads();
    }
    cluster_sync_all();   // neither CTA releases shared memory or TMEM the other may still touch
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc_pair(tmem_base, 512);
    }
}

template <int MODE, int D, int ABFMT, typename OutT>
int launch_chunk_pair_one(const PassParams& p, int in_dtype, cudaStream_t st) {
    using C = CpCfg<D>;
    CUtensorMap mx, myh, mz, ms, mo;
    int rc;
    constexpr bool STATE_MN = (MODE == FWDC || MODE == DVC);
    constexpr int out_dtype = sizeof(OutT) == 4 ? MLSTM_DT_F32 : (ABFMT == 1 ? MLSTM_DT_BF16 : MLSTM_DT_F16);
    // staging rows of 128 bytes: the 128-byte swizzle of the operand maps; of 64 bytes: the output maps
    rc = sizeof(OutT) == 4 && C::STAGE_ROW == 128 ? tc_make_map(&mo, p.out, p.BH, p.S, D, out_dtype, false, 32)
                                                  : tc_make_map_out(&mo, p.out, p.BH, p.S, D, out_dtype, 32);
    if (rc != MLSTM_OK) return rc;
    if ((rc = tc_make_map(&mx, p.X, p.BH, p.S, D, in_dtype, false, 128)) != MLSTM_OK) return rc;
    if ((rc = tc_make_map(&myh, p.Y, p.BH, p.S, D, in_dtype, false, 64)) != MLSTM_OK) return rc;
    if ((rc = tc_make_map(&mz, p.Z, p.BH, p.S, D, in_dtype, false, 128)) != MLSTM_OK) return rc;
    if ((rc = tc_make_map(&ms, p.states, p.BH * p.NB * (p.state_parts == 2 ? 2 : 1), D, D, in_dtype, false, STATE_MN ? 128 : D / 2)) != MLSTM_OK) return rc;
    auto kern = mlstm_chunk_pair<MODE, D, ABFMT, OutT>;
    {   // the shared-memory opt-in is a per-device property of the kernel: set once per device
        static std::atomic<bool> opted[64];
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return MLSTM_E_CUDA;
        if (!opted[dev].load(std::memory_order_acquire)) {
            cudaFuncAttributes fa;
            cudaError_t ce = cudaFuncGetAttributes(&fa, kern);
            if (ce == cudaSuccess && !register_split_fits(fa.numRegs)) ce = cudaErrorLaunchOutOfResources;
            if (ce != cudaSuccess) {
                cudaGetLastError();
                return note_cuda_error(ce, "registers of mlstm_chunk_pair at launch against its register split");
            }
            ce = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES);
            if (ce != cudaSuccess) {
                cudaGetLastError();
                return note_cuda_error(ce, "cudaFuncSetAttribute(MaxDynamicSharedMemorySize)");
            }
            opted[dev].store(true, std::memory_order_release);
        }
    }
    const int NT = p.Spad / TILE;
    const long long total = static_cast<long long>((NT + 1) / 2) * p.BH;
    if (total > 0x3fffffffLL) return MLSTM_E_SHAPE;
    const int sms = tc_sm_count();
    if (sms < 2) return MLSTM_E_CUDA;
    // persistent pairs with equal shares; the grid does not have to be resident at once: CTAs only wait inside their pair
    const unsigned npairs = static_cast<unsigned>(total < sms / 2 ? total : sms / 2);
    cudaError_t ce = launch_pdl(kern, dim3(2 * npairs), dim3(NTHREADS), C::SMEM_BYTES, st, mx, myh, mz, ms, mo, p);
    if (ce != cudaSuccess) cudaGetLastError();
    return ce == cudaSuccess ? MLSTM_OK : note_cuda_error(ce, "launch of mlstm_chunk_pair");
}

// fp16: the output pass and DVC, which the chunkwise entry points use; DQC and DKC serve the bf16 route alone (mm_chunk_route)
template <int MODE, int D>
int launch_chunk_pair_fmt(const PassParams& p, int in_dtype, int out_dtype, cudaStream_t st) {
    if (in_dtype == MLSTM_DT_BF16) {
        if (out_dtype == in_dtype) return launch_chunk_pair_one<MODE, D, 1, __nv_bfloat16>(p, in_dtype, st);
        if constexpr (MODE == FWDC)
            if (out_dtype == MLSTM_DT_F32) return launch_chunk_pair_one<MODE, D, 1, float>(p, in_dtype, st);
    } else if constexpr (MODE == DQC || MODE == DKC) {
        return MLSTM_E_UNSUPPORTED;
    } else if (in_dtype == MLSTM_DT_F16) {
        if (out_dtype == in_dtype) return launch_chunk_pair_one<MODE, D, 0, __half>(p, in_dtype, st);
        if constexpr (MODE == FWDC)
            if (out_dtype == MLSTM_DT_F32) return launch_chunk_pair_one<MODE, D, 0, float>(p, in_dtype, st);
    }
    return MLSTM_E_ARG;
}

template <int MODE>
int launch_chunk_pair_d(const PassParams& p, int in_dtype, int out_dtype, cudaStream_t st) {
    return p.D == 128 ? launch_chunk_pair_fmt<MODE, 128>(p, in_dtype, out_dtype, st)
                      : launch_chunk_pair_fmt<MODE, 256>(p, in_dtype, out_dtype, st);
}

}  // namespace

bool chunk_pair_supported(int D, int in_dtype, int chunk_tiles) {
    return (D == 128 || D == 256) && (in_dtype == MLSTM_DT_F16 || in_dtype == MLSTM_DT_BF16) && chunk_tiles % 2 == 0;
}

int launch_chunk_pair(int mode, const PassParams& p, int in_dtype, int out_dtype, cudaStream_t st) {
    if (!chunk_pair_supported(p.D, in_dtype, p.chunk_tiles)) return MLSTM_E_UNSUPPORTED;
    if (!p.An_bound || !p.states || p.NB <= 0) return MLSTM_E_ARG;
    switch (mode) {
        case FWDC: return p.zstate ? launch_chunk_pair_d<FWDC>(p, in_dtype, out_dtype, st) : MLSTM_E_ARG;
        case DQC: return p.zstate ? launch_chunk_pair_d<DQC>(p, in_dtype, out_dtype, st) : MLSTM_E_ARG;
        case DKC: return p.rvec ? launch_chunk_pair_d<DKC>(p, in_dtype, out_dtype, st) : MLSTM_E_ARG;
        case DVC: return launch_chunk_pair_d<DVC>(p, in_dtype, out_dtype, st);
    }
    return MLSTM_E_UNSUPPORTED;
}

}  // namespace mlstm

extern "C" int mlstm_selftest_register_split(int registers_per_thread) {
    return mlstm::register_split_fits(registers_per_thread) ? MLSTM_OK : MLSTM_E_CUDA;
}
