// fp64_gemm.cu -- native FP64 GEMM for sm_100a on the FP64 tensor-core path (DMMA).
//
// Replaces the arithmetic of MGXBench's sharedABMultiply / sharedABMultiplyAccumulate
// (1D-row-block/mulmat_kernel.cu:39-80 and 100-142): C = A*B, or C += (A*B summed over the chunk).
//
// The kernel is bound by the FP64 tensor pipe (64 FMA per clock and SM, 37.2 TFLOP/s on 148 SMs at
// 1965 MHz); the design keeps the four sub-partitions of all SMs equally busy.
//   * Work is cut in units of 8 columns of a 64-row band.  Every sub-partition owns 16 rows of the
//     band and all of the tile's columns, so a tile of any width up to 128 columns loads the four
//     pipes equally and its time is proportional to its width (a last band of up to 32 rows is
//     spread over them by columns, see COST).  The CTAs' shares of a product can then
//     be equal to within one unit (Walk), whatever the shape; fp64_cut.h has the cut.  Against whole
//     128 x 128 tiles dealt to the SMs: N = 256 (4 tiles on 148 SMs) 39 -> 7.6 us a call, N = 1024 (64
//     tiles) 145 -> 68 us, 1024 x 4096 x 2048 (256 tiles: 1.73 waves paid as 2) 614 -> 483 us, N = 8192
//     35.1 -> 36.6 TFLOP/s.
//   * warpgroup 0 (producer, one lane): TMA 2D loads of A (BM x 32 doubles) and B (32 x up to 128)
//     into a ring of 128-byte swizzled tiles, each stage guarded by a full/empty mbarrier pair.  No
//     multicast.  Operands TMA cannot describe (odd leading dimension or K offset, unaligned
//     base) are first re-laid into stream-ordered scratch by pack_kernel.
//   * warpgroups 1-4 (consumers): four warps per sub-partition, each 16 rows x a quarter of the
//     tile's units as DMMA m16n8k8 accumulators (up to 4).  With two warps of up to 8 units the
//     pipe waited on fragment loads and stage hand-offs 5.6% of the time (ncu): 2048 x 8192 x 8192
//     ran at 35.3, with three warps at 35.5, with four at 35.8 TFLOP/s.  128-row bands (half the
//     A fragment loads per MMA) reached 35.7 and cut ragged shapes more coarsely.
//   * The reduction index is permuted inside every group of 8 (physical order 0,1,4,5 | 2,3,6,7)
//     identically for A and B, so each fragment load from the swizzled tiles hits every shared
//     memory bank exactly twice (the minimum for 256 bytes).
//   * Epilogue: C = acc (beta 0) or C = C + acc (beta 1), one rounding, as the reference.
// An element's reduction runs over K in the same order whatever the tile width or the share it falls
// in, so the cut does not change a bit of the result.
#include <atomic>
#include <chrono>
#include <climits>
#include <cstdio>
#include <cstring>
#include <type_traits>

#include "fp64_cut.h"
#include "mgx_common.cuh"

namespace mgx {
namespace fp64 {

constexpr int SUB_WARPS = CWARPS / 4;                     // consumer warps of a sub-partition
constexpr int WARP_UNITS = (TILE_UNITS + SUB_WARPS - 1) / SUB_WARPS;  // units of a consumer warp
constexpr int PRODUCER_WARPS = 4;                         // one warpgroup
constexpr int THREADS = (CWARPS + PRODUCER_WARPS) * 32;   // 640 = 5 warpgroups
// Register split (setmaxnreg): the block launches with 640 x 96 registers; the producer warpgroup
// gives back down to 32 each and the four consumer warpgroups take 112 each:
// 128 x 32 + 512 x 112 = 61440 = 640 x 96.  The host refuses to launch unless the compiled
// kernel has exactly LAUNCH_REGS registers per thread, so the split always adds up.
constexpr int LAUNCH_REGS = 96, PRODUCER_REGS = 32, CONSUMER_REGS = 112;
static_assert(CWARPS == 16 && BM == 64, "the warps' split of a tile");
static_assert(PRODUCER_WARPS * 32 * PRODUCER_REGS + CWARPS * 32 * CONSUMER_REGS == THREADS * LAUNCH_REGS,
              "register split must equal the launch budget");

// Shared memory: A as two boxes of 64 rows x 16 doubles, B as up to eight boxes of 32 rows x 16
// doubles; 4 stages of 48 KiB.
constexpr int A_BOX_BYTES = BM * 128;
constexpr int B_BOX_BYTES = BK * 128;
constexpr int A_STAGE_BYTES = 2 * A_BOX_BYTES;
constexpr int STAGE_BYTES = A_STAGE_BYTES + 8 * B_BOX_BYTES;
constexpr int STAGES = 4;
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 256;

struct Params : Cut {
    double *C;
    int m, n;
    int a_x0;         // first column of A (k_offset)
    int ldc;
    int beta_one;     // 1: C + A B, 0: A B, -1: 0 + A B (no negative zeros)
    int vec_store;    // C rows 16-byte aligned (ldc even, C aligned)
    int *status;
    int panel_kb;       // > 0: SUMMA panels of so many K blocks; the running sum takes each panel's product
                        // with one rounding
    unsigned long long *sk_tickets;  // stream-K: one arrival ticket per tile and consumer warp
    unsigned long long sk_epoch;     // stream-K: this launch's ticket tag (a ticket of another tag counts 0)
    double *sk_partial; // stream-K: two partial accumulators per CTA (its first and last segment)
    double *partial;    // split-K: slice s of the product goes to partial + s * partial_stride
    int partial_ld;     // even, so the partial rows are 16-byte aligned
    size_t partial_stride;
};

// Stream-K tickets: (launch tag << 8) | arrivals.  A ticket written by an earlier launch (another
// tag), or never written, counts as no arrivals, so nothing clears the tickets before a launch.
// Arrivals per tile are at most the grid size, below 256.
__device__ __forceinline__ int ticket_count(unsigned long long *tk, unsigned long long tag)
{
    const unsigned long long v = atomicAdd(tk, 0ull);
    return (v >> 8) == tag ? (int)(v & 255u) : 0;
}

// Takes a ticket; returns the arrivals before this one.  The first to arrive replaces what an earlier launch left
// by this launch's tag and no arrivals; only this launch's warps write here now, so whoever loses that
// exchange finds the tag set, and each arrival is one addition.  (As one compare-and-swap per arrival,
// all but one of the CTAs that arrive together failed each time and tried again: 128 x 128 x 4096, 74
// pieces a tile, 81 us, 43 now.)
__device__ __forceinline__ int ticket_take(unsigned long long *tk, unsigned long long tag, int *status)
{
    const unsigned long long old = atomicAdd(tk, 0ull);
    if ((old >> 8) != tag) atomicCAS(tk, old, tag << 8);
    const unsigned long long prev = atomicAdd(tk, 1ull);
    if ((prev >> 8) == tag) return (int)(prev & 255u);
    record_status(status, kDevTicket);  // another launch uses the workspace at the same time
    return -1;
}

// Waits for a stage on behalf of the whole warp; false when the bounded wait ran out.
__device__ __forceinline__ bool warp_wait(uint64_t *bar, uint32_t parity, int lane, int *status, int code)
{
    if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
    int got = 1;
    if (lane == 0) got = mbar_wait_bounded(bar, parity, status, code);
    got = __shfl_sync(0xffffffffu, got, 0);
    // every lane observes the completed phase itself, so its reads of the stage are ordered after it
    return got && mbar_try_wait(bar, parity);
}

// Position of a consumer warp in the ring and its constant address parts.
struct Consumer {
    uint64_t *full, *empty;
    uint32_t smem_base;
    int lane, strip, u_first;
    int stage;
    uint32_t phase;
};

// A warp's reduction of one item: NU units (from its first unit of the tile) over K blocks
// [kb_begin, kb_end).  PANELS: after every panel the accumulators are added to tot with
// one rounding and cleared, as the reference's C += panel product does.
template <int NU, bool PANELS>
__device__ __forceinline__ bool reduce_item(const Params &p, Consumer &c, int kb_begin, int kb_end,
                                            double (&acc)[WARP_UNITS][4], double (&tot)[PANELS ? WARP_UNITS : 1][4])
{
    const int g = c.lane >> 2, t = c.lane & 3;
    // One m16n8k8 per unit: logical k t -> physical k (t&1) + 4(t>>1), logical t+4 -> the same plus 2,
    // i.e. the permutation 0,1,4,5 | 2,3,6,7 of the group of 8.  With the 128-byte swizzle, an odd
    // group of 8 k (A) or an odd unit (B) flips bit 6 of the address, so two offsets per step serve
    // the whole stage; the rest are constants.
    const uint32_t a0 = (uint32_t)((c.strip * 16 + g) * 128 + ((((t >> 1) * 2) ^ g) << 4) + ((t & 1) << 3));
    const uint32_t a1 = a0 ^ 16u;
    uint32_t b_off[2][2];
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
        for (int step = 0; step < 2; ++step) {
            const int unit = c.u_first + e, phys = (t & 1) + ((t >> 1) << 2) + 2 * step;
            b_off[e][step] = (uint32_t)(A_STAGE_BYTES + (unit >> 1) * B_BOX_BYTES + phys * 128 +
                                        ((((unit & 1) * 4 + (g >> 1)) ^ phys) << 4) + ((g & 1) << 3));
        }
    int panel_left = PANELS ? p.panel_kb : 0;
    for (int kb = kb_begin; kb < kb_end; ++kb) {
        if (!warp_wait(&c.full[c.stage], c.phase, c.lane, p.status, kDevTimeoutFull)) return false;
        const uint32_t base = c.smem_base + c.stage * STAGE_BYTES;
#pragma unroll
        for (int kb8 = 0; kb8 < (NU > 0 ? 4 : 0); ++kb8) {
            const uint32_t flip = (kb8 & 1) * 64u, abox = base + (kb8 >> 1) * A_BOX_BYTES;
            const double af[4] = {lds_f64(abox + (a0 ^ flip)), lds_f64(abox + (a0 ^ flip) + 1024),
                                  lds_f64(abox + (a1 ^ flip)), lds_f64(abox + (a1 ^ flip) + 1024)};
            double bf[NU > 0 ? NU : 1][2];
#pragma unroll
            for (int step = 0; step < 2; ++step)
#pragma unroll
                for (int u = 0; u < NU; ++u)
                    bf[u][step] = lds_f64(base + b_off[u & 1][step] + (u >> 1) * B_BOX_BYTES + kb8 * 1024);
#pragma unroll
            for (int u = 0; u < NU; ++u) dmma_16x8x8(acc[u], af, bf[u]);
        }
        __syncwarp();
        if (c.lane == 0) mbar_arrive(&c.empty[c.stage]);
        if (++c.stage == STAGES) {
            c.stage = 0;
            c.phase ^= 1u;
        }
        if constexpr (PANELS) {
            if (--panel_left == 0 || kb + 1 == kb_end) {
                panel_left = p.panel_kb;
#pragma unroll
                for (int u = 0; u < NU; ++u)
#pragma unroll
                    for (int v = 0; v < 4; ++v) {
                        tot[u][v] = __dadd_rn(tot[u][v], acc[u][v]);
                        acc[u][v] = 0.0;
                    }
            }
        }
    }
    return true;
}

// A kernel for each form, so that each is scheduled for itself: with stream-K's epilogue in the whole-K
// kernel 2048 x 8192 x 2048 took 1930 us against 1885, N = 1024 68.5 against 66.8, N = 256 5.04 against 4.77.
template <bool PANELS, bool STREAMK>
__global__ void __launch_bounds__(THREADS, 1)
    dgemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, Params p)
{
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                                            ~uintptr_t(1023));
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + STAGES * STAGE_BYTES);
    uint64_t *empty = full + STAGES;

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], CWARPS);
        }
        fence_barrier_init();
    }
    if (warp == 0 && lane == 0) {
        tma_prefetch_desc(&tmA);
        tma_prefetch_desc(&tmB);
    }
    __syncthreads();
    // Launched as a programmatic dependent: everything above overlapped the previous kernel in the
    // stream; nothing below reads or writes memory before that kernel has finished.  The next
    // kernel may be scheduled now (it cannot share an SM with this one, and waits the same way).
    pdl_wait();
    pdl_trigger();

    // The panel form's two accumulator sets leave it few registers, and its speed depends on what else is
    // live: 3001 x 5002 x 4096 in panels of 512 takes 3496 us with 64-bit positions, 3565 with 32-bit
    // ones.  The whole-K form is 1.5% faster with 32-bit ones at N = 256.
    Walk<STREAMK, std::conditional_t<PANELS || STREAMK, long long, unsigned>> walk;
    walk.init(p, blockIdx.x, gridDim.x);
    Item it;

    if (warp < PRODUCER_WARPS) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(PRODUCER_REGS));
        if (threadIdx.x != 0) return;
        // ------------------------------------------------------------ TMA producer (one lane)
        int stage = 0;
        uint32_t phase = 0;
        int armed_parity[STAGES];
        for (int s = 0; s < STAGES; ++s) armed_parity[s] = -1;
        bool ok = true;
        while (ok && walk.next(p, it)) {
            const int m0 = it.band * BM, n0 = it.u0 * UNIT;
            const int boxes = (it.units + 1) >> 1;
            for (int kb = it.kb_begin; kb < it.kb_end; ++kb) {
                if (!mbar_wait_bounded(&empty[stage], phase ^ 1u, p.status, kDevTimeoutEmpty)) {
                    ok = false;
                    break;
                }
                unsigned char *sA = smem + stage * STAGE_BYTES;
                unsigned char *sB = sA + A_STAGE_BYTES;
                const int k0 = kb * BK;
                mbar_arrive_expect_tx(&full[stage], A_STAGE_BYTES + boxes * B_BOX_BYTES);
                armed_parity[stage] = (int)phase;
                tma_load_2d(sA, &tmA, p.a_x0 + k0, m0, &full[stage]);
                tma_load_2d(sA + A_BOX_BYTES, &tmA, p.a_x0 + k0 + 16, m0, &full[stage]);
                for (int j = 0; j < boxes; ++j) tma_load_2d(sB + j * B_BOX_BYTES, &tmB, n0 + 16 * j, k0, &full[stage]);
                if (++stage == STAGES) {
                    stage = 0;
                    phase ^= 1u;
                }
            }
        }
        // Never leave the CTA with a tensor copy still writing its shared memory.
        for (int s = 0; s < STAGES; ++s)
            if (armed_parity[s] >= 0) mbar_wait_bounded(&full[s], (uint32_t)armed_parity[s], p.status, kDevTimeoutFull);
        return;
    }

    // ---------------------------------------------------------------- consumers
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(CONSUMER_REGS));
    const int cw = warp - PRODUCER_WARPS;
    const int g = lane >> 2;
    const int t = lane & 3;
    Consumer c;
    c.full = full;
    c.empty = empty;
    c.smem_base = smem_u32(smem);
    c.lane = lane;
    c.stage = 0;
    c.phase = 0;

    // dst (+)= acc for this lane's fragments, masked to C's bounds (dst = C, or a split-K slice of
    // the partial products).
    auto store_acc = [&](const double (&acc)[WARP_UNITS][4], int nu, int beta_one, double *dst_base, int ld,
                         int vec_store) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int row = it.band * BM + c.strip * 16 + h * 8 + g;
            if (row >= p.m) continue;
            double *crow = dst_base + (size_t)row * ld;
#pragma unroll
            for (int u = 0; u < WARP_UNITS; ++u) {
                const int col = (it.u0 + c.u_first + u) * UNIT + 2 * t;
                if (u >= nu || col >= p.n) break;
                double v0 = acc[u][2 * h], v1 = acc[u][2 * h + 1];
                if (vec_store && col + 1 < p.n) {
                    double2 *dst = reinterpret_cast<double2 *>(crow + col);
                    if (beta_one) {
                        const double2 old = *dst;
                        v0 = old.x + v0;
                        v1 = old.y + v1;
                    }
                    *dst = make_double2(v0, v1);
                } else {
                    crow[col] = beta_one ? crow[col] + v0 : v0;
                    if (col + 1 < p.n) crow[col + 1] = beta_one ? crow[col + 1] + v1 : v1;
                }
            }
        }
    };

    while (walk.next(p, it)) {
        if (PANELS) it.strips = 2;  // (a variable one costs 1%; make_cut asks for no other)
        int nu;
        warp_part(it, cw, c.strip, c.u_first, nu);

        double acc[WARP_UNITS][4];
        double tot[PANELS ? WARP_UNITS : 1][4];
#pragma unroll
        for (int j = 0; j < WARP_UNITS; ++j)
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                acc[j][v] = 0.0;
                if (PANELS) tot[PANELS ? j : 0][v] = 0.0;
            }

        bool ok = true;
        // the unit count as a constant, so that its fragments and accumulators stay in registers
        switch (nu) {
        case 0: ok = reduce_item<0, PANELS>(p, c, it.kb_begin, it.kb_end, acc, tot); break;
        case 1: ok = reduce_item<1, PANELS>(p, c, it.kb_begin, it.kb_end, acc, tot); break;
        case 2: ok = reduce_item<2, PANELS>(p, c, it.kb_begin, it.kb_end, acc, tot); break;
        case 3: ok = reduce_item<3, PANELS>(p, c, it.kb_begin, it.kb_end, acc, tot); break;
        default: ok = reduce_item<WARP_UNITS, PANELS>(p, c, it.kb_begin, it.kb_end, acc, tot); break;
        }
        if (!ok) return;
        if constexpr (PANELS) {
#pragma unroll
            for (int j = 0; j < WARP_UNITS; ++j)
#pragma unroll
                for (int v = 0; v < 4; ++v) acc[j][v] = tot[j][v];
        }
        if constexpr (STREAMK) {
            // A tile whose K range spans several CTAs' shares is finished by the CTA that
            // arrives last at its ticket: every piece's accumulator goes to that CTA's partial
            // slot, and the last arrival adds the pieces in K order (p0 + p1) + p2 ... and
            // stores C.  No CTA waits for another.
            if (it.kb_begin == 0 && it.kb_end == p.kblocks) {
                store_acc(acc, nu, p.beta_one, p.C, p.ldc, p.vec_store);
            } else {
                // (only here: its 64-bit divisions take longer than a tile of one K block.  1102 x 19749 x 3:
                // 119 us with them for every tile, 70 without)
                const Piece q = piece_of(p, it, blockIdx.x, gridDim.x);
                const int pieces = q.pieces, j = q.index;
                // Each consumer warp owns the same fragment of the tile in every piece, so it
                // finishes that fragment on its own: a ticket per (tile, warp), and no barrier
                // between the warps (a warp that gave up on a wait cannot block the others).
                constexpr int NACC = WARP_UNITS * 4;
                constexpr size_t PART = (size_t)CWARPS * 32 * NACC;  // doubles per partial slot
                const int ct = threadIdx.x - PRODUCER_WARPS * 32;     // consumer thread 0..511
                double(&af)[NACC] = reinterpret_cast<double(&)[NACC]>(acc);
                const int na = nu * 4;
                unsigned long long *ticket = p.sk_tickets + (size_t)it.tile * CWARPS + cw;
                // The head piece is usually computed last (at the end of its CTA's share):
                // when every later piece has taken its ticket, it finishes the tile without
                // writing its own partial.
                int last = 0;
                if (j == 0) {
                    if (lane == 0) last = ticket_count(ticket, p.sk_epoch) == pieces - 1;
                    last = __shfl_sync(0xffffffffu, last, 0);
                }
                if (!last) {
                    double *mine = p.sk_partial + ((size_t)blockIdx.x * 2 + q.slot) * PART;
#pragma unroll
                    for (int i = 0; i < NACC; ++i)
                        if (i < na) __stcg(mine + (size_t)i * (CWARPS * 32) + ct, af[i]);
                    __threadfence();
                    __syncwarp();
                    if (lane == 0) last = ticket_take(ticket, p.sk_epoch, p.status) == pieces - 1;
                    last = __shfl_sync(0xffffffffu, last, 0);
                }
                if (last) {
                    __threadfence();
                    // Bound by the trips to L2, one after the other because the pieces add up in order: 32
                    // loads are in flight at a time, two units of four pieces.  One by one, behind a test for the
                    // own piece (which has been written too, unless it is the first and never left its
                    // registers), 128 x 128 x 4096 with 74 pieces took 335 us against 82, 256^3 with 8 35 against 15.
                    constexpr int TRIP = 4;
#pragma unroll
                    for (int i0 = 0; i0 < NACC; i0 += 8) {
                        if (i0 >= na) break;
                        if (j > 0) {
                            const double *p0 = p.sk_partial + ((size_t)q.c0 * 2 + q.slot0) * PART + ct;
#pragma unroll
                            for (int i = 0; i < 8; ++i) af[i0 + i] = __ldcg(p0 + (i0 + i) * (CWARPS * 32));
                        }
                        for (int jj = 1; jj < pieces; jj += TRIP) {
                            double v[TRIP][8];
#pragma unroll
                            for (int r = 0; r < TRIP; ++r) {
                                // pieces after the first start their CTA's share: slot 0
                                const double *pr = p.sk_partial + (size_t)(q.c0 + min(jj + r, pieces - 1)) * 2 * PART + ct;
#pragma unroll
                                for (int i = 0; i < 8; ++i) v[r][i] = __ldcg(pr + (i0 + i) * (CWARPS * 32));
                            }
#pragma unroll
                            for (int r = 0; r < TRIP; ++r)
                                if (jj + r < pieces) {
#pragma unroll
                                    for (int i = 0; i < 8; ++i) af[i0 + i] = af[i0 + i] + v[r][i];
                                }
                        }
                    }
                    store_acc(acc, nu, p.beta_one, p.C, p.ldc, p.vec_store);
                    // a graph replays the launch with the same tag, which must find no arrivals
                    if (lane == 0) atomicExch(ticket, 0ull);
                }
            }
        } else if (p.ksplit > 1) {
            store_acc(acc, nu, 0, p.partial + (size_t)it.slice * p.partial_stride, p.partial_ld, 1);
        } else {
            // 0 + the sum changes no value but -0.0, and integer instructions tell that one: an addition would
            // wait for the FP64 pipe behind the other warps' products (1000 x 9000 x 512 266 us without, 267
            // so, 274 with additions).  The panel form's running sum starts from zero by itself.
            if (!PANELS && p.beta_one < 0) {
#pragma unroll
                for (int j = 0; j < WARP_UNITS; ++j)
#pragma unroll
                    for (int v = 0; v < 4; ++v)
                        if (__double_as_longlong(acc[j][v]) == LLONG_MIN) acc[j][v] = 0.0;
            }
            store_acc(acc, nu, p.beta_one > 0, p.C, p.ldc, p.vec_store);
        }
    }
}

// Split-K epilogue: C = (beta ? C : 0) + (slice 0 + slice 1 + ...), the slices summed in that
// fixed order, so the result does not depend on which CTA finished first.  Two columns per
// thread: the partial rows are 16-byte aligned (even ld, 256-byte aligned base; the pad column
// of an odd n is read and dropped).
__global__ void splitk_reduce(double *__restrict__ C, int ldc, int beta_one, const double *__restrict__ P, int ld,
                              size_t stride, int slices, int m, int n)
{
    const bool c_vec = ((ldc & 1) == 0) && ((reinterpret_cast<uintptr_t>(C) & 15) == 0);
    for (int row = blockIdx.x; row < m; row += gridDim.x) {
        const double *prow = P + (size_t)row * ld;
        double *crow = C + (size_t)row * ldc;
        for (int col = 2 * threadIdx.x; col < n; col += 2 * blockDim.x) {
            double2 v = *reinterpret_cast<const double2 *>(prow + col);
            int s = 1;
            for (; s + 3 < slices; s += 4) {  // four independent loads in flight, summed in order
                const double2 p1 = *reinterpret_cast<const double2 *>(prow + (size_t)s * stride + col);
                const double2 p2 = *reinterpret_cast<const double2 *>(prow + (size_t)(s + 1) * stride + col);
                const double2 p3 = *reinterpret_cast<const double2 *>(prow + (size_t)(s + 2) * stride + col);
                const double2 p4 = *reinterpret_cast<const double2 *>(prow + (size_t)(s + 3) * stride + col);
                v.x = (((v.x + p1.x) + p2.x) + p3.x) + p4.x;
                v.y = (((v.y + p1.y) + p2.y) + p3.y) + p4.y;
            }
            for (; s < slices; ++s) {
                const double2 p1 = *reinterpret_cast<const double2 *>(prow + (size_t)s * stride + col);
                v.x += p1.x;
                v.y += p1.y;
            }
            if (col + 1 < n) {
                if (c_vec) {
                    double2 *dst = reinterpret_cast<double2 *>(crow + col);
                    if (beta_one) {
                        const double2 o = *dst;
                        v.x = o.x + v.x;
                        v.y = o.y + v.y;
                    }
                    *dst = v;
                } else {
                    crow[col] = beta_one ? crow[col] + v.x : v.x;
                    crow[col + 1] = beta_one ? crow[col + 1] + v.y : v.y;
                }
            } else {
                crow[col] = beta_one ? crow[col] + v.x : v.x;
            }
        }
    }
}

// One operand re-laid with an even pitch and a 16-byte aligned base; live columns, the rest zero.
struct Pack {
    const double *src;
    double *dst;
    int rows, cols, live, ld_src;  // destination pitch (even), live columns, source pitch
    int log2_width;                // threads of a row: 2^log2_width, each PACK_PER columns
    int chunks;                    // column chunks of a row
    unsigned blocks;
};
constexpr int PACK_THREADS = 256, PACK_PER = 8;

// Both operands in one launch: blocks [0, a.blocks) pack A, the others B; a block packs one column chunk
// of PACK_THREADS >> log2_width rows, the narrowest power of two of threads that a row's columns keep
// busy (a block for each row however short: 2,000,000 rows of 3 took as many blocks).  Bound by
// memory: 8-byte accesses because an odd pitch allows no wider ones, eight in flight per thread (a
// grid-stride loop with a 64-bit division per element took 42 us for 98 MB, this takes 26).
__global__ void __launch_bounds__(PACK_THREADS) pack_kernel(const Pack a, const Pack b)
{
    const bool is_a = blockIdx.x < a.blocks;
    const Pack &q = is_a ? a : b;
    const unsigned i = is_a ? blockIdx.x : blockIdx.x - a.blocks;
    const int width = 1 << q.log2_width;
    const long long r = (long long)(i / q.chunks) * (PACK_THREADS >> q.log2_width) + (threadIdx.x >> q.log2_width);
    if (r >= q.rows) return;
    const int c0 = (int)(i % q.chunks) * (width * PACK_PER) + (threadIdx.x & (width - 1));
    const double *src = q.src + r * q.ld_src;
    double *dst = q.dst + r * q.cols;
    double v[PACK_PER];
#pragma unroll
    for (int u = 0; u < PACK_PER; ++u) {
        const int c = c0 + u * width;
        v[u] = c < q.live ? __ldg(src + c) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < PACK_PER; ++u) {
        const int c = c0 + u * width;
        if (c < q.cols) dst[c] = v[u];
    }
}

}  // namespace fp64
}  // namespace mgx

using namespace mgx;

// Split-K geometry: K blocks per slice and the number of non-empty slices for `ksplit` asked.
static void splitk_geometry(int k_len, int ksplit, int *kb_split, int *slices)
{
    const int kblocks = (k_len + fp64::BK - 1) / fp64::BK;
    if (ksplit < 1) ksplit = 1;
    if (ksplit > kblocks) ksplit = kblocks > 0 ? kblocks : 1;
    *kb_split = (kblocks + ksplit - 1) / ksplit;
    *slices = *kb_split > 0 ? (kblocks + *kb_split - 1) / *kb_split : 1;
}

// Launches the split-K epilogue (also used by the Ozaki form's split-K).
int mgx_launch_splitk_reduce(double *C, int ldc, int beta_one, const double *P, int ld, size_t stride, int slices,
                             int m, int n, cudaStream_t stream)
{
    if (m <= 0 || n <= 0) return MGX_SUCCESS;
    int rgrid = mgx_sm_count() * 8;
    if (rgrid > m) rgrid = m;
    fp64::splitk_reduce<<<rgrid, 256, 0, stream>>>(C, ldc, beta_one, P, ld, stride, slices, m, n);
    MGX_HOST_CHECK(cudaGetLastError());
    return MGX_SUCCESS;
}

size_t mgx_fp64_splitk_bytes(int m, int n, int k, int ksplit)
{
    int kbs, slices;
    splitk_geometry(k, ksplit, &kbs, &slices);
    if (slices <= 1 || m <= 0 || n <= 0) return 0;
    return (size_t)slices * (size_t)m * (size_t)((n + 1) & ~1) * sizeof(double) + 256;
}

// Stream-K workspace: two partial accumulators (64 x 128 doubles) per CTA of the grid, then one 8-byte
// ticket per tile and consumer warp.
static size_t streamk_partial_bytes(int grid)
{
    return (size_t)grid * 2 * fp64::CWARPS * 32 * fp64::WARP_UNITS * 4 * sizeof(double);
}

size_t mgx_fp64_streamk_bytes(int m, int n, int k)
{
    if (m <= 0 || n <= 0 || k <= 0) return 0;
    const fp64::Cut c = fp64::shape_cut(m, n, k);
    const size_t tiles = (size_t)c.bands * c.tiles_n;
    return streamk_partial_bytes(fp64::streamk_grid(c, mgx_sm_count())) +
           ((tiles * fp64::CWARPS * sizeof(unsigned long long) + 255) & ~size_t(255));
}

// A fresh ticket tag per stream-K launch, 56 bits.  Odd, so that cleared memory reads as no arrivals, and
// counted from a start that differs from process to process: the workspace is the caller's, never cleared,
// and small tags would be found in what other programs leave in memory, such as an array of indices.
static unsigned long long streamk_tag()
{
    static std::atomic<unsigned long long> next{[] {
        // splitmix64 (Steele, Lea and Flood 2014) of the time and of an address of this process
        unsigned long long z = (unsigned long long)std::chrono::high_resolution_clock::now().time_since_epoch().count();
        z ^= (unsigned long long)reinterpret_cast<uintptr_t>(&z) << 20;
        z += 0x9e3779b97f4a7c15ull;
        z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
        z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
        return z ^ (z >> 31);
    }()};
    return (next.fetch_add(2, std::memory_order_relaxed) | 1ull) & ((1ull << 56) - 1);
}

// How launch_dgemm cuts and accumulates a product (the defaults: one whole-K product).
struct DgemmMode {
    int panel_k = 0;   // > 0: SUMMA panels of this width, a multiple of 32
    int ksplit = 1;    // K slices
    int streamk = 0;
    void *ws = nullptr;
    size_t ws_bytes = 0;
};

static int launch_dgemm(const double *A, const double *B, double *C, int m, int n, int k_len, int a_x0, int a_x_end,
                        int b_rows, int lda, int ldb, int ldc, int beta_one, cudaStream_t stream, const DgemmMode &mode)
{
    if (m <= 0 || n <= 0) return MGX_SUCCESS;
    if (k_len <= 0) {
        if (beta_one > 0) return MGX_SUCCESS;
        // C = A*B with an empty reduction is zero
        MGX_HOST_CHECK(cudaMemset2DAsync(C, (size_t)ldc * sizeof(double), 0, (size_t)n * sizeof(double), m, stream));
        return MGX_SUCCESS;
    }
    const bool panels = mode.panel_k > 0 && mode.panel_k < k_len;
    int slices = 1, kb_split = 0, grid = 0;
    splitk_geometry(k_len, panels ? 1 : mode.ksplit, &kb_split, &slices);
    fp64::Params p;
    memset(&p, 0, sizeof p);
    static_cast<fp64::Cut &>(p) =
        fp64::make_cut(m, n, k_len, slices, kb_split,
                       panels         ? fp64::CutMode::kPanels
                       : mode.streamk ? fp64::CutMode::kStreamK
                                      : fp64::CutMode::kWhole,
                       mgx_sm_count(), &grid);
    p.C = C;
    p.m = m;
    p.n = n;
    p.ldc = ldc;
    p.beta_one = beta_one;
    p.vec_store = ((ldc & 1) == 0) && ((reinterpret_cast<uintptr_t>(C) & 15) == 0);
    p.status = mgx_device_status_ptr();
    if (panels) p.panel_kb = mode.panel_k / fp64::BK;
    p.partial_ld = (n + 1) & ~1;
    p.partial_stride = (size_t)m * (size_t)p.partial_ld;
    if (slices > 1) {
        const size_t need = (size_t)slices * p.partial_stride * sizeof(double);
        if (!mode.ws || mode.ws_bytes < need || (reinterpret_cast<uintptr_t>(mode.ws) & 255)) {
            mgx_set_last_message("FP64 split-K: workspace of %zu bytes (aligned to 256) needed, %zu given", need,
                                 mode.ws_bytes);
            return MGX_E_WORKSPACE;
        }
        p.partial = reinterpret_cast<double *>(mode.ws);
    }

    if (mode.streamk) {
        if (grid > 255) {  // arrivals per tile must fit a ticket's 8-bit count
            mgx_set_last_message("FP64 stream-K: grid of %d CTAs exceeds 255", grid);
            return MGX_E_UNSUPPORTED;
        }
        const size_t pbytes = streamk_partial_bytes(grid);
        const size_t tbytes = (size_t)p.bands * p.tiles_n * fp64::CWARPS * sizeof(unsigned long long);
        if (!mode.ws || mode.ws_bytes < pbytes + tbytes || (reinterpret_cast<uintptr_t>(mode.ws) & 255)) {
            mgx_set_last_message("FP64 stream-K: workspace of %zu bytes (aligned to 256) needed, %zu given",
                                 pbytes + tbytes, mode.ws_bytes);
            return MGX_E_WORKSPACE;
        }
        p.sk_partial = reinterpret_cast<double *>(mode.ws);
        p.sk_tickets = reinterpret_cast<unsigned long long *>(reinterpret_cast<char *>(mode.ws) + pbytes);
        p.sk_epoch = streamk_tag();
    }

    // TMA wants 16-byte aligned bases, pitches and (even) columns; operands that are not so are
    // packed first.  Where no column of A is to be read (a chunk wholly beyond k_total) its map
    // lies wholly left of the columns asked for, so every box is zero fill.
    const bool a_none = a_x_end <= a_x0;
    if (a_none) {
        A = reinterpret_cast<const double *>(reinterpret_cast<uintptr_t>(A) & ~uintptr_t(15));
        lda = a_x_end = 2;
        a_x0 = fp64::BK;
    }
    const bool a_ok = ((reinterpret_cast<uintptr_t>(A) & 15) == 0) && lda % 2 == 0 && a_x0 % 2 == 0;
    const bool b_ok = ((reinterpret_cast<uintptr_t>(B) & 15) == 0) && ldb % 2 == 0;
    char *scratch = nullptr;
    if (!a_ok || !b_ok) {
        const int lda2 = (k_len + 1) & ~1, ldb2 = (n + 1) & ~1;
        const size_t abytes = a_ok ? 0 : ((size_t)m * lda2 * sizeof(double) + 255) & ~size_t(255);
        const size_t bbytes = b_ok ? 0 : (size_t)b_rows * ldb2 * sizeof(double);
        const int arc = mgx_scratch_alloc(reinterpret_cast<void **>(&scratch), abytes + bbytes + 256, stream);
        if (arc != MGX_SUCCESS) return arc;
        auto pack = [](const double *src, char *dst, int rows, int cols, int live, int ld) {
            fp64::Pack q = {src, reinterpret_cast<double *>(dst), rows, cols, live, ld, 0, 0, 0u};
            while ((fp64::PACK_PER << q.log2_width) < cols && (1 << q.log2_width) < fp64::PACK_THREADS) ++q.log2_width;
            const int chunk = fp64::PACK_PER << q.log2_width, per = fp64::PACK_THREADS >> q.log2_width;
            q.chunks = (cols - 1) / chunk + 1;
            q.blocks = (unsigned)((rows - 1) / per + 1) * (unsigned)q.chunks;
            return q;
        };
        fp64::Pack qa = {}, qb = {};
        if (!a_ok) {
            qa = pack(A + a_x0, scratch, m, lda2, a_x_end - a_x0, lda);
            A = qa.dst;
            lda = lda2;
            a_x0 = 0;
            a_x_end = k_len;
        }
        if (!b_ok) {
            qb = pack(B, scratch + abytes, b_rows, ldb2, n, ldb);
            B = qb.dst;
            ldb = ldb2;
        }
        fp64::pack_kernel<<<qa.blocks + qb.blocks, fp64::PACK_THREADS, 0, stream>>>(qa, qb);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) {
            mgx_set_last_cuda_error(e, "operand packing", __FILE__, __LINE__);
            cudaFreeAsync(scratch, stream);
            return MGX_E_CUDA;
        }
    }
    p.a_x0 = a_x0;
    CUtensorMap tmA, tmB;
    int rc = mgx_encode_tmap_2d(&tmA, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 8, A, (uint64_t)a_x_end, (uint64_t)m,
                                (uint64_t)lda * 8, 16, fp64::BM, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc == MGX_SUCCESS)
        rc = mgx_encode_tmap_2d(&tmB, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 8, B, (uint64_t)n, (uint64_t)b_rows,
                                (uint64_t)ldb * 8, 16, fp64::BK, CU_TENSOR_MAP_SWIZZLE_128B);
    auto launch = [&](auto kernel) -> int {
        cudaFuncAttributes fa;
        MGX_HOST_CHECK(cudaFuncGetAttributes(&fa, kernel));
        if (fa.numRegs != fp64::LAUNCH_REGS) {
            mgx_set_last_message("FP64 kernel compiled with %d registers/thread, expected %d for its register split",
                                 fa.numRegs, fp64::LAUNCH_REGS);
            return MGX_E_UNSUPPORTED;
        }
        MGX_HOST_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, fp64::SMEM_BYTES));
        // the set-up above the kernel's wait overlaps the end of the previous kernel in the stream
        MGX_HOST_CHECK(mgx_launch_dependent(kernel, dim3((unsigned)grid), dim3(fp64::THREADS), fp64::SMEM_BYTES, stream,
                                            tmA, tmB, p));
        return MGX_SUCCESS;
    };
    if (rc == MGX_SUCCESS) rc = panels           ? launch(fp64::dgemm_kernel<true, false>)
                                : mode.streamk ? launch(fp64::dgemm_kernel<false, true>)
                                               : launch(fp64::dgemm_kernel<false, false>);
    if (scratch) cudaFreeAsync(scratch, stream);
    if (rc != MGX_SUCCESS) return rc;
    MGX_HOST_CHECK(cudaGetLastError());
    if (slices > 1)
        return mgx_launch_splitk_reduce(C, ldc, beta_one, p.partial, p.partial_ld, p.partial_stride, slices, m, n,
                                        stream);
    return MGX_SUCCESS;
}

// C (+)= A[:, a_x0 : a_x0 + k_len] * B[0 : k_len, :] with the library's FP64 kernel.
// a_x_end: A columns at or beyond it read as zero; b_rows: rows of B that exist.  beta_one: 1 adds to C, 0
// writes the product, -1 writes 0 + the product (the first of several panels).
int mgx_launch_dgemm(const double *A, const double *B, double *C, int m, int n, int k_len, int a_x0, int a_x_end,
                     int b_rows, int lda, int ldb, int ldc, int beta_one, cudaStream_t stream)
{
    return launch_dgemm(A, B, C, m, n, k_len, a_x0, a_x_end, b_rows, lda, ldb, ldc, beta_one, stream, DgemmMode{});
}

// SUMMA: C = 0 + the sum over the panels of width panel_k (a multiple of 32, or all of K) of A B, each
// panel's product added with one rounding.
int mgx_launch_dgemm_panels(const double *A, const double *B, double *C, int m, int n, int k, int lda, int ldb,
                            int ldc, int panel_k, cudaStream_t stream)
{
    DgemmMode mode;
    mode.panel_k = panel_k;
    return launch_dgemm(A, B, C, m, n, k, 0, k, k, lda, ldb, ldc, -1, stream, mode);
}

// Split-K form: the K range is cut into `ksplit` slices whose products land in `partial`
// (mgx_fp64_splitk_bytes bytes, 256-byte aligned) and are summed into C in slice order by a second
// kernel.
int mgx_launch_dgemm_splitk(const double *A, const double *B, double *C, int m, int n, int k, int lda, int ldb,
                            int ldc, int beta_one, int ksplit, void *partial, size_t partial_bytes,
                            cudaStream_t stream)
{
    DgemmMode mode;
    mode.ksplit = ksplit;
    mode.ws = partial;
    mode.ws_bytes = partial_bytes;
    return launch_dgemm(A, B, C, m, n, k, 0, k, k, lda, ldb, ldc, beta_one, stream, mode);
}

// Stream-K form over 64-row tiles: every CTA takes an equal share of all tiles' K blocks.
int mgx_launch_dgemm_streamk(const double *A, const double *B, double *C, int m, int n, int k, int lda, int ldb,
                             int ldc, int beta_one, void *workspace, size_t workspace_bytes, cudaStream_t stream)
{
    DgemmMode mode;
    mode.streamk = 1;
    mode.ws = workspace;
    mode.ws_bytes = workspace_bytes;
    return launch_dgemm(A, B, C, m, n, k, 0, k, k, lda, ldb, ldc, beta_one, stream, mode);
}
