// Role-specialised paired step kernel: the tiled step with its filters, its collisions and its
// copies in warps of their own.
//
// Same step as stream_collide (C/evolution.h:358-684) for FP32 arithmetic with FP32, FP16 or BF16
// population storage, two spanwise-adjacent nodes per thread and every FP32 operation packed across
// the pair, as step_pair.cu. There one thread filters, combines and collides its node pair, eight
// warps per SM (tensor memory holds no more rings) take the same steps at the same time, and every
// plane waits for a CTA barrier: 42% of the issue slots were used. Here a CTA of 640 threads owns a
// tile of 512 nodes (TY = 512/NX full rows), one CTA per SM, and four kinds of warps run at
// their own pace, coupled by mbarriers only:
//   * the front producer copies the planes of a wall-normal segment into the front stages
//     (populations 3, 4, 7..10, 15..18 with three halo rows on each side; 5, 6, 11..14), the target
//     producer the target planes' populations 0, 1, 2 and xi weights into target stages, each as 4D
//     tensor-map boxes (tiles whose halo wraps around the period: row runs);
//   * eight filter warps (two per tensor-memory lane quarter) filter a plane: four take the
//     populations that need one axis (y: 3, 4, 15..18, x: 11..14; raw 5, 6), four the ones that need
//     both (7..10). A thread takes the same node pair of two adjacent rows, so the eight halo rows
//     it reads serve two 7-row sums (a row pair costs 80 shared loads instead of 140), and
//     writes both rows' values into a ring of eight planes in tensor memory (2 rows x 8 planes
//     x 32 columns = all 512 columns of the SM);
//   * eight collide warps (two per lane quarter, one per row of the pair) combine seven planes of
//     the ring along xi, apply walls and BFL rows, collide the pair and store it. Populations 1 and 2
//     need no xi filter and come from the target stage, so the ring needs no delay line.
// Tiles are four rows high at NX = 128 instead of two: 2.5 instead of 4 halo rows are copied per row.
#pragma once

#include <cstring>
#include <type_traits>

#include "pair_math.cuh"
#include "step_common.cuh"
#include "step_launch.hpp"
#include "step_tiled.hpp"
#include "pair_helpers.cuh"
#include "tile_helpers.cuh"
#include "step_roles.hpp"

namespace islbm {

namespace {

constexpr int COLLIDE_WARPS = 8, FILTER_WARPS = 8;
constexpr int COLLIDE_THREADS = 32*COLLIDE_WARPS;
constexpr int FILTER_WARP0 = COLLIDE_WARPS, FRONT_WARP = FILTER_WARP0 + FILTER_WARPS, TARGET_WARP = FRONT_WARP + 1;
constexpr int THREADS = 640;          // five warpgroups: collide, collide, row filter, quad filter, producers
constexpr int ACTIVE_THREADS = 32*(TARGET_WARP + 1);
// registers per thread of the warpgroups after the split: two collide groups, row filter, quad filter,
// producers, together at most the 5*96 that the CTA is launched with
// (16-bit formats, LES, 128x256x192: 152/72/72 205.9 us per step, 144/80/80 217.6, 160/64/64 207.4)
template <class S> struct Regs { static constexpr int collide = 152, rows = 72, quads = 72, copies = 32; };
template <> struct Regs<float> { static constexpr int collide = 152, rows = 80, quads = 64, copies = 32; };
constexpr int SLOTS = 8;              // ring planes

// named barriers: 1 collide warps, 2 work item (batched kernel), 3, 4 filter row groups, 5 end of the
// ring's use (filter warps arrive, collide warps wait)
constexpr int BAR_COLLIDE = 1, BAR_ITEM = 2, BAR_FILTER = 3, BAR_RING_END = 5;
constexpr int RING_THREADS = 32*(COLLIDE_WARPS + FILTER_WARPS);

template <int R> __device__ __forceinline__ void regs_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(R)); }
template <int R> __device__ __forceinline__ void regs_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(R)); }
__device__ __forceinline__ void bar_sync(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int threads) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
// D3Q19 streamwise component of e_q (C/initialization.h:7-12 ordering)
__host__ __device__ constexpr int ey_of(int q) {
    return (q == 3 || q == 7 || q == 8 || q == 15 || q == 17) ? 1 : (q == 4 || q == 9 || q == 10 || q == 16 || q == 18) ? -1 : 0;
}
// populations of a front stage in order: 3, 4, 7..10, 15..18 (with halo rows), 5, 6, 11..14
__host__ __device__ constexpr int FQ(int i) {
    return i < 2 ? 3 + i : i < 6 ? 5 + i : i < 10 ? 9 + i : i < 12 ? i - 5 : i - 1;
}

// Shared-memory layout of one tile (compile-time offsets):
//   NFS front stages; NTS target stages (populations 0, 1, 2 as TY rows, then the rows' duplicated
//   xi weights, TY x 128 floats); ybuf [2][TY][2][NX/2] float4: streamwise-filtered (7, 8, 9, 10)
//   by plane parity, the even and the odd node of each pair apart (consecutive threads, consecutive
//   16 bytes); a double2 of sums per collide thread; near wall rows: one sum per collide
//   thread, their weights, lists of two planes; mbarriers; timeout flag and TMEM address.
template <class S, int NXC>
struct RLay {
    static constexpr int NX = NXC, PR = NX/2, TY = 512/NX;
    static constexpr int EB = (int)sizeof(S);
    static constexpr int up128(int v) { return (v + 127)/128*128; }
    static constexpr int row = NX*EB;
    static constexpr int halo_pop = (TY + 6)*row, plain_pop = TY*row;
    static constexpr int f_off(int i) { return i < 10 ? i*halo_pop : up128(10*halo_pop) + (i - 10)*plain_pop; }
    static constexpr int front_bytes = up128(f_off(16));
    static constexpr unsigned front_tx = (unsigned)(10*halo_pop + 6*plain_pop);
    static constexpr int w_off = up128(3*plain_pop);
    static constexpr int target_bytes = w_off + TY*512;
    static constexpr unsigned target_tx = (unsigned)(3*plain_pop + TY*512);
    static constexpr int ybuf_bytes = 2*512*16, sums_bytes = COLLIDE_THREADS*16;
    static constexpr int mids_bytes = 512*4, near_bytes = 2*(1 + 2*TY)*4 + TY*4;
    // front stages: as many as fit, up to three. The copies of a plane take about 2.5 us from issue to
    // completion under load, longer than a plane's work: with two stages the copies' latency set
    // the pace (FP32 256x128x192 without collisions and stores 184 us per step, with them 207)
    static constexpr int room = 227*1024 - ybuf_bytes - sums_bytes - mids_bytes - near_bytes - 1024;
    static constexpr int fit = (room - 2*target_bytes)/front_bytes;
    static constexpr int NFS = fit > 3 ? 3 : fit;
    static constexpr int NTS = NFS*front_bytes + 4*target_bytes <= room ? 4 : 2;
    static_assert(NFS >= 2, "two front stages");
    static constexpr int target_off = NFS*front_bytes;
    static constexpr int ybuf_off = target_off + NTS*target_bytes;
    static constexpr int sums_off = ybuf_off + ybuf_bytes;
    static constexpr int mids_off = sums_off + sums_bytes, wz_off = mids_off + mids_bytes, near_off = wz_off + TY*4;
    static constexpr int bar_off = (wz_off + near_bytes + 7)/8*8;
    // mbarriers: front full, front empty, target full, target empty, ring full and ring free per
    // lane quarter and slot
    static constexpr int B_FF = 0, B_FE = NFS, B_TF = 2*NFS, B_TE = B_TF + NTS, B_RF = B_TE + NTS, B_RE = B_RF + 4*SLOTS;
    static constexpr int NBARS = B_RE + 4*SLOTS;
    static constexpr int flag_off = bar_off + NBARS*8;
    // one CTA per SM: its ring takes all 512 tensor-memory columns
    static constexpr int smem_bytes = flag_off + 16 > 152*1024 ? flag_off + 16 : 152*1024;
    static_assert(smem_bytes <= 227*1024, "layout exceeds shared memory");
};

struct RoleTM {
    CUtensorMap m[5];
};

template <class S, bool LES, int NXC>
struct RoleKernel {
    using LY = RLay<S, NXC>;
    static constexpr int NX = NXC, PR = LY::PR, TY = LY::TY;
    static_assert(2*Regs<S>::collide + Regs<S>::rows + Regs<S>::quads + Regs<S>::copies <= 480, "register split");
    struct Scal { float f6, f12, rho_mod, tau, lesC; };
    const S *fo;
    S *fn;
    S *fnq[19];                // fn + q*N
    Tables<float> T;
    StepConst k;
    TiledConst tc;
    Ctrl *ctrl;
    float *rho_out, *u_out, *v_out, *w_out;
    int macros_on, mass_on;
    unsigned seat_set;         // seats of this launch

    // position in a ring of N stages: index and phase parity
    template <int N> struct Stage {
        int i = 0;
        unsigned ph = 0;
        __device__ __forceinline__ void next() { if (++i == N) { i = 0; ph ^= 1u; } }
    };
    struct Piece {
        int y0, yskip, ta, tb, p0, p1;   // first row, rows done by the previous tile, targets, planes
    };
    __device__ __forceinline__ int window_base(int t) const { return t <= 3 ? 0 : (t >= k.NZ - 4 ? k.NZ - 7 : t - 3); }
    // the last tile of a streamwise count that is no multiple of TY starts at NY - TY and skips the
    // rows that the previous tile owns
    __device__ __forceinline__ Piece make_piece(int tile, int ta, int tb) const {
        Piece P;
        P.y0 = min(tile*TY, k.NY - TY);
        P.yskip = tile*TY - P.y0;
        P.ta = ta;
        P.tb = tb;
        P.p0 = window_base(ta);
        P.p1 = window_base(tb - 1) + 6;
        return P;
    }
    // The work items of a CTA: M = zmain*tiles long segments, one for each of the first M CTAs, and
    // the rest of every column in zrest equal segments for the others (see split_columns)
    template <class F>
    __device__ __forceinline__ void for_items(int seat, F &&f) const {
        const int tiles = (k.NY + TY - 1)/TY, M = tc.zmain*tiles, b = seat;
        if (b < M) {
            const int seg = b/tiles;
            f(make_piece(b - seg*tiles, seg*tc.zlen, (seg + 1)*tc.zlen));
            return;
        }
        const int z0 = tc.zmain*tc.zlen, nz = k.NZ - z0;
        for (int j = b - M; j < tiles*tc.zsegs; j += (int)gridDim.x - M) {
            const int seg = j/tiles;
            f(make_piece(j - seg*tiles, z0 + seg*nz/tc.zsegs, z0 + (seg + 1)*nz/tc.zsegs));
        }
    }

    // Wait for a phase of mbarrier b: no sleep between the tries (sleeping poll loops wake up late; FP32
    // 217 instead of 207 us per step with them). Bounded: after about two seconds, or once another
    // thread of the CTA has given up, the thread stops waiting for good; the step then ends with
    // ctrl->fault set.
    __device__ __forceinline__ void wait(unsigned char *smem, int b, unsigned parity, bool &faulted) const {
        if (faulted) return;
        uint64_t *bar = (uint64_t *)(smem + LY::bar_off) + b;
        if (mbar_try_wait(bar, parity)) return;
        volatile int *flag = (volatile int *)(smem + LY::flag_off);
        const unsigned long long t0 = global_ns();
        do {
#pragma unroll 1
            for (int i = 0; i < 64; i++)
                if (mbar_try_wait(bar, parity)) return;
        } while (!*flag && global_ns() - t0 < 2000000000ULL);
        faulted = true;
        *flag = 1;
        atomicOr(&ctrl->fault, 1u);
    }
    __device__ __forceinline__ uint64_t *bars(unsigned char *smem, int b) const { return (uint64_t *)(smem + LY::bar_off) + b; }

    // ---- producers (one lane each) ----

    __device__ __forceinline__ void produce_front(unsigned char *smem, const Piece &P, Stage<LY::NFS> &at, unsigned &count, bool &faulted,
                                                  const CUtensorMap *tm) const {
        const int NY = k.NY;
        const size_t N = (size_t)NX*NY*k.NZ;
        constexpr int rows = TY + 6;
        const bool boxes = tm && P.y0 >= 3 && P.y0 + TY + 3 <= NY;
        for (int p = P.p0; p <= P.p1; p++, count++, at.next()) {
            const int st = at.i;
            wait(smem, LY::B_FE + st, at.ph ^ 1u, faulted);   // (at once in the first round)
            if (faulted || *(volatile int *)(smem + LY::flag_off)) return;   // no further copies after a timeout
            if (p == k.drill_plane) continue;                                // failure drill: this plane never arrives
            uint64_t *bar = bars(smem, LY::B_FF + st);
            unsigned char *dst = smem + st*LY::front_bytes;
            mbar_expect_tx(bar, LY::front_tx);
            if (boxes) {
                tma_load4(dst + LY::f_off(0), tm + 0, 0, P.y0 - 3, p, 3, bar);
                tma_load4(dst + LY::f_off(2), tm + 1, 0, P.y0 - 3, p, 7, bar);
                tma_load4(dst + LY::f_off(6), tm + 1, 0, P.y0 - 3, p, 15, bar);
                tma_load4(dst + LY::f_off(10), tm + 2, 0, P.y0, p, 5, bar);
                tma_load4(dst + LY::f_off(12), tm + 3, 0, P.y0, p, 11, bar);
            } else {
                // row runs: a halo that wraps around the period is two runs per population. Compile-time
                // operands: a loop took 140 cycles per copy, and the wrapping tiles twice the others' time
                const S *plane = fo + (size_t)p*NY*NX;
                const int ys = P.y0 >= 3 ? P.y0 - 3 : P.y0 - 3 + NY;
                const unsigned first = (unsigned)min(rows, NY - ys)*LY::row, rest = (unsigned)LY::halo_pop - first;
                const S *a = plane + (size_t)ys*NX;
#pragma unroll
                for (int i = 0; i < 10; i++) bulk_g2s(dst + i*LY::halo_pop, a + (size_t)FQ(i)*N, first, bar);
                if (rest)
#pragma unroll
                    for (int i = 0; i < 10; i++) bulk_g2s(dst + i*LY::halo_pop + first, plane + (size_t)FQ(i)*N, rest, bar);
                if (tm) {
                    tma_load4(dst + LY::f_off(10), tm + 2, 0, P.y0, p, 5, bar);
                    tma_load4(dst + LY::f_off(12), tm + 3, 0, P.y0, p, 11, bar);
                } else {
#pragma unroll
                    for (int i = 10; i < 16; i++)
                        bulk_g2s(dst + LY::f_off(i), plane + (size_t)FQ(i)*N + (size_t)P.y0*NX, LY::plain_pop, bar);
                }
            }
        }
    }

    __device__ __forceinline__ void produce_targets(unsigned char *smem, const Piece &P, Stage<LY::NTS> &at, unsigned &count, bool &faulted,
                                                    const CUtensorMap *tm) const {
        const int NY = k.NY;
        const size_t N = (size_t)NX*NY*k.NZ;
        for (int t = P.ta; t < P.tb; t++, count++, at.next()) {
            const int st = at.i;
            wait(smem, LY::B_TE + st, at.ph ^ 1u, faulted);
            if (faulted || *(volatile int *)(smem + LY::flag_off)) return;
            uint64_t *bar = bars(smem, LY::B_TF + st);
            unsigned char *dst = smem + LY::target_off + st*LY::target_bytes;
            mbar_expect_tx(bar, LY::target_tx);
            if (tm) tma_load4(dst, tm + 4, 0, P.y0, t, 0, bar);
            else
#pragma unroll 1
                for (int q = 0; q < 3; q++)
                    bulk_g2s(dst + q*LY::plain_pop, fo + (size_t)q*N + ((size_t)t*NY + P.y0)*NX, LY::plain_pop, bar);
            bulk_g2s(dst + LY::w_off, T.wxi2 + ((size_t)t*NY + P.y0)*128, (unsigned)(TY*512), bar);
        }
    }

    // A producer's end: bounded wait for its last copies, so that none is in flight when the CTA
    // exits (in a healthy run the consumers have waited for every one already)
    __device__ __forceinline__ void drain(unsigned char *smem, int bar0, int stages, unsigned count) const {
        for (unsigned c = count > (unsigned)stages ? count - stages : 0; c < count; c++) {
            bool done = false;
            for (int it = 0; it < (1 << 22) && !done; ++it) {
                done = mbar_try_wait(bars(smem, bar0 + (int)(c % stages)), (c/stages) & 1u);
                if (!done && it > 32) {
                    if (*(volatile int *)(smem + LY::flag_off) && it > (1 << 12)) break;   // never issued (after a timeout)
                    __nanosleep(256);
                }
            }
        }
    }

    // ---- filter warps ----

    // A thread of a filter warp (lane quarter w) takes the node pair (x0, x0 + 1) of rows r0, r0 + 1.
    // The streamwise sums of population FQ(q) for both rows from the eight halo rows
    template <int Q0, int NQ>
    __device__ __forceinline__ void y_filter(const S *base, V2 (&acc)[2][NQ]) const {
        for (int q = 0; q < NQ; q++) acc[0][q] = acc[1][q] = V2(0.f);
#pragma unroll
        for (int b = 0; b < 8; b++) {
#pragma unroll
            for (int q = 0; q < NQ; q++) {
                const V2 f = ld2v<S>(base + LY::f_off(Q0 + q)/LY::EB + b*NX);
                const int set = ey_of(FQ(Q0 + q)) > 0 ? 0 : 1;
                if (b < 7) acc[0][q] = V2(tc.wyb[set][b])*f + acc[0][q];
                if (b > 0) acc[1][q] = V2(tc.wyb[set][b - 1])*f + acc[1][q];
            }
        }
    }
    // the ring slot is free once both collide warps of this lane quarter are done with its plane
    __device__ __forceinline__ void wait_slot(unsigned char *smem, unsigned seq, int w, bool &faulted) const {
        wait(smem, LY::B_RE + w*SLOTS + (int)(seq % SLOTS), (seq/SLOTS & 1u) ^ 1u, faulted);
        tmem_fence_after();
    }
    __device__ __forceinline__ void filtered(unsigned char *smem, int st, unsigned seq, int w, int lane) const {
        tmem_wait_st();
        tmem_fence_before();
        __syncwarp();
        if (lane == 0) {
            mbar_arrive(bars(smem, LY::B_FE + st));                                // front stage read
            mbar_arrive(bars(smem, LY::B_RF + w*SLOTS + (int)(seq % SLOTS)));      // ring columns written
        }
    }

    // Row filter warps: y filter of 3, 4, 15..18, raw 5, 6 and x filter of 11..14
    __device__ __forceinline__ void filter_rows(unsigned char *smem, const Stage<LY::NFS> &at, unsigned seq, int w, int lane, uint32_t tl, bool &faulted) const {
        const int i = 32*w + lane, r0 = 2*(i/PR), j = i % PR, x0 = 2*j;
        const unsigned char *front = smem + at.i*LY::front_bytes;
        const uint32_t col = tl + 32u*(seq % SLOTS);
        wait(smem, LY::B_FF + at.i, at.ph, faulted);
        float o[2][8];
#pragma unroll
        for (int r = 0; r < 2; r++)
#pragma unroll
            for (int q = 0; q < 4; q++)
                x_filter((const S *)(front + LY::f_off(12 + q)) + (r0 + r)*NX, j, q & 1, o[r][2*q], o[r][2*q + 1]);
        const S *base = (const S *)front + r0*NX + x0;
        V2 a[2][2], b[2][4];
        y_filter<0, 2>(base, a);
        y_filter<6, 4>(base, b);
        wait_slot(smem, seq, w, faulted);
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const V2 r5 = ld2v<S>((const S *)(front + LY::f_off(10)) + (r0 + r)*NX + x0);
            const V2 r6 = ld2v<S>((const S *)(front + LY::f_off(11)) + (r0 + r)*NX + x0);
            const V2 p[8] = {a[r][0], a[r][1], r5, r6, b[r][0], b[r][1], b[r][2], b[r][3]};
            float v[16];
#pragma unroll
            for (int q = 0; q < 8; q++) { v[2*q] = p[q].v.x; v[2*q + 1] = p[q].v.y; }
            tmem_st16(col + 256u*r, v);
            tmem_st8(col + 256u*r + 24u, o[r][0], o[r][1], o[r][2], o[r][3], o[r][4], o[r][5], o[r][6], o[r][7]);
        }
        filtered(smem, at.i, seq, w, lane);
    }

    // Quad filter warps: y and x filter of 7, 8, 9, 10, the y-filtered values of a node as one quad in ybuf
    __device__ __forceinline__ void filter_quads(unsigned char *smem, const Stage<LY::NFS> &at, unsigned seq, int w, int lane, uint32_t tl, bool &faulted) const {
        const int i = 32*w + lane, g = i/PR, r0 = 2*g, j = i % PR, x0 = 2*j;
        const unsigned char *front = smem + at.i*LY::front_bytes;
        float4 *yb = (float4 *)(smem + LY::ybuf_off) + (seq & 1u)*512 + r0*NX;   // [row][parity][pair]
        const uint32_t col = tl + 32u*(seq % SLOTS) + 16u;
        wait(smem, LY::B_FF + at.i, at.ph, faulted);
        {
            V2 acc[2][4];
            y_filter<2, 4>((const S *)front + r0*NX + x0, acc);
#pragma unroll
            for (int r = 0; r < 2; r++) {
                yb[r*NX + j] = make_float4(acc[r][0].v.x, acc[r][1].v.x, acc[r][2].v.x, acc[r][3].v.x);
                yb[r*NX + PR + j] = make_float4(acc[r][0].v.y, acc[r][1].v.y, acc[r][2].v.y, acc[r][3].v.y);
            }
        }
        // the row pair's quads are complete (the buffer of the plane after next is this one again:
        // every thread has read it by the next plane's barrier)
        if constexpr (PR > 32) bar_sync(BAR_FILTER + g, PR);
        else __syncwarp();
        float o[2][8];
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const float4 *ev = yb + r*NX, *od = ev + PR;
            float4 gv[8];
#pragma unroll
            for (int a = 0; a < 8; a++) gv[a] = (a & 1) ? ev[(j - 1 + a/2) & (PR - 1)] : od[(j - 2 + a/2) & (PR - 1)];
            // (7, 8) and (9, 10) of node 0 / node 1
            V2 n0a = V2(tc.wx[0])*V2(gv[0].x, gv[0].y), n0b = V2(tc.wx[0])*V2(gv[0].z, gv[0].w);
            V2 n1a = V2(tc.wx[0])*V2(gv[1].x, gv[1].y), n1b = V2(tc.wx[0])*V2(gv[1].z, gv[1].w);
#pragma unroll
            for (int a = 1; a < 7; a++) {
                const V2 wv = V2(tc.wx[a]);
                n0a = wv*V2(gv[a].x, gv[a].y) + n0a;
                n0b = wv*V2(gv[a].z, gv[a].w) + n0b;
                n1a = wv*V2(gv[a + 1].x, gv[a + 1].y) + n1a;
                n1b = wv*V2(gv[a + 1].z, gv[a + 1].w) + n1b;
            }
            o[r][0] = n0a.v.x; o[r][1] = n1a.v.x; o[r][2] = n0a.v.y; o[r][3] = n1a.v.y;
            o[r][4] = n0b.v.x; o[r][5] = n1b.v.x; o[r][6] = n0b.v.y; o[r][7] = n1b.v.y;
        }
        wait_slot(smem, seq, w, faulted);
#pragma unroll
        for (int r = 0; r < 2; r++)
            tmem_st8(col + 256u*r, o[r][0], o[r][1], o[r][2], o[r][3], o[r][4], o[r][5], o[r][6], o[r][7]);
        filtered(smem, at.i, seq, w, lane);
    }
    __device__ __forceinline__ void filter_planes(unsigned char *smem, const Piece &P, Stage<LY::NFS> &at, unsigned &seq, int warp, int lane,
                                                  uint32_t tl, bool &faulted) const {
        const int planes = P.p1 - P.p0 + 1;
        if (warp < 4)
#pragma unroll 1
            for (int i = 0; i < planes; i++, seq++, at.next()) filter_rows(smem, at, seq, warp, lane, tl, faulted);
        else
#pragma unroll 1
            for (int i = 0; i < planes; i++, seq++, at.next()) filter_quads(smem, at, seq, warp - 4, lane, tl, faulted);
    }

    // Spanwise filter of one population (set 0: departure x - minSize, 1: x + minSize) for the node
    // pair 2j, 2j + 1 of a row, from aligned node pairs L[k] = (v[x0+k], v[x0+k+1]), k = -4, -2, .., 4:
    // node 0 sums w[k+3] v[x0+k] + w[k+4] v[x0+k+1], node 1 w[k+2] v[x0+k] + w[k+3] v[x0+k+1], each
    // split over the two lanes of its accumulator (odd and even stencil points). The two single-lane
    // end terms are separate products, so that no zero weight multiplies a value outside a node's
    // stencil, and both nodes add the same terms in the same order.
    __device__ __forceinline__ void x_filter(const S *row, int j, int set, float &o0, float &o1) const {
        V2 L[5];
#pragma unroll
        for (int kk = 0; kk < 5; kk++) L[kk] = ld2v<S>(row + 2*((j - 2 + kk) & (PR - 1)));
        V2 a0 = V2(0.f, tc.wxa[set][0].y*L[0].v.y), a1 = V2(tc.wxb[set][0])*L[1];
#pragma unroll
        for (int kk = 1; kk < 4; kk++) {
            a0 = V2(tc.wxa[set][kk])*L[kk] + a0;
            if (kk < 3) a1 = V2(tc.wxb[set][kk])*L[kk + 1] + a1;
        }
        a1.v.x = __fmaf_rn(tc.wxb[set][3].x, L[4].v.x, a1.v.x);
        o0 = a0.v.x + a0.v.y;
        o1 = a1.v.x + a1.v.y;
    }

    // ---- collide warps ----

    // xi combination of the seven ring planes seq .. seq + 6 with the duplicated-pair xi weights of
    // the target row w (7 x 16 floats: (xi3, xi3, xi4, xi4, xi5, xi5, xi6, xi6, xi15, xi15, ...,
    // xi18, xi18) per stencil point). Writes F[3..18].
    // `under`: work done while the first two planes' loads are under way.
    template <class U>
    __device__ __forceinline__ void xi_combine(uint32_t tl, unsigned seq, const float4 *w, V2 (&F)[19], U &&under) const {
        V2 acc[16];
        auto add = [&](const uint32_t (&g)[32], int c) {
            float4 wq[4];
#pragma unroll
            for (int m = 0; m < 4; m++) wq[m] = w[4*c + m];
            const V2 x3(wq[0].x, wq[0].y), x4(wq[0].z, wq[0].w), x5(wq[1].x, wq[1].y), x6(wq[1].z, wq[1].w);
            const V2 x15(wq[2].x, wq[2].y), x16(wq[2].z, wq[2].w), x17(wq[3].x, wq[3].y), x18(wq[3].z, wq[3].w);
            // slot order 3, 4, 5, 6, 15, 16, 17, 18, 7, 8, 9, 10, 11, 12, 13, 14
            const V2 wj[16] = {x3, x4, x5, x6, x15, x16, x17, x18, x3, x3, x4, x4, x5, x5, x6, x6};
#pragma unroll
            for (int q = 0; q < 16; q++) {
                const V2 v(__uint_as_float(g[2*q]), __uint_as_float(g[2*q + 1]));
                if (c == 0) acc[q] = wj[q]*v;
                else acc[q] = wj[q]*v + acc[q];
            }
        };
#pragma unroll
        for (int c = 0; c < 7; c += 2) {
            uint32_t g0[32], g1[32];
            tmem_ld32(tl + 32u*((seq + c) % SLOTS), g0);
            if (c < 6) tmem_ld32(tl + 32u*((seq + c + 1) % SLOTS), g1);
            if (c == 0) under();
            tmem_wait_ld();
            tmem_tie(g0);
            add(g0, c);
            if (c < 6) {
                tmem_tie(g1);
                add(g1, c + 1);
            }
        }
        constexpr int RQ[16] = {3, 4, 5, 6, 15, 16, 17, 18, 7, 8, 9, 10, 11, 12, 13, 14};
#pragma unroll
        for (int q = 0; q < 16; q++) F[RQ[q]] = acc[q];
    }

    __device__ __forceinline__ float bw(int s, int a, int idx) const {
        const int nb = 2*k.NYD6;
        return idx < nb ? __ldg(T.bfl_w + ((size_t)s*7 + a)*nb + idx) : 0.f;
    }
    // Sums of the opposite populations for wall distances below one half, in the order of the paired and
    // gather kernels (x innermost, then y, then xi): FP16 storage carries a changed last place on, and
    // 2,000 steps over the steep hill (alpha 0.73, whose first rows are such) made 9e-4 of it.
    // y and xi only (populations without an x axis):
    __device__ __forceinline__ V2 bfl_y_xi(int q, int yset, int zset, int x0, int y, int r, int iy) const {
        const size_t N = (size_t)NX*k.NY*k.NZ;
        V2 g = V2(0.f);
#pragma unroll 1
        for (int c = 0; c < 7; c++) {
            V2 in = V2(0.f);
#pragma unroll
            for (int b = 0; b < 7; b++) in = V2(bw(yset, b, iy))*ld2g<S>(fo + q*N + bfl_row(c, y - 3 + b) + x0, q) + in;
            g = V2(bw(zset, c, r))*in + g;
        }
        return g;
    }
    // x and y at plane c: a node pair's stencils are five aligned pairs of every row (all loads first: they are one
    // latency)
    __device__ __forceinline__ V2 bfl_x_y(int q, int c, int xset, int yset, int x0, int y, int r, int iy) const {
        const S *plane = fo + q*((size_t)NX*k.NY*k.NZ);
        V2 f[7][5], wx[7], mid = V2(0.f);
        float wy[7];
        int x[5];
#pragma unroll
        for (int m = 0; m < 5; m++) x[m] = (x0 - 4 + 2*m) & (NX - 1);
#pragma unroll
        for (int b = 0; b < 7; b++) {
            const S *p = plane + (unsigned)bfl_row(c, y - 3 + b);
#pragma unroll
            for (int m = 0; m < 5; m++) f[b][m] = ld2g<S>(p + x[m], q);
        }
#pragma unroll
        for (int a = 0; a < 7; a++) {   // reference: X weights at [i], Y weights at [j]
            wx[a] = V2(bw(xset, a, k.bfl_mode ? r : x0 + 3), bw(xset, a, k.bfl_mode ? r : x0 + 4));
            wy[a] = bw(yset, a, iy);
        }
#pragma unroll
        for (int b = 0; b < 7; b++) {
            V2 in = V2(0.f);
#pragma unroll
            for (int a = 0; a < 7; a++)
                in = wx[a]*((a & 1) ? f[b][(a + 1)/2] : V2(f[b][a/2].v.y, f[b][a/2 + 1].v.x)) + in;
            mid = V2(wy[b])*in + mid;
        }
        return mid;
    }
    __device__ __forceinline__ size_t bfl_row(int c, int yy) const {
        const int NY = k.NY;
        yy = yy < 0 ? yy + NY : (yy >= NY ? yy - NY : yy);
        return ((size_t)c*NY + yy)*NX;
    }

    // One flag type of the BFL rows (C/evolution.h:505-572) of a whole row y at plane z <= 1. dst / src:
    // populations set and their opposites, the first without and the other two with an x filter (N3 = 1
    // or 3). Returns 0 where the row is not set, 1 with the populations (full values) in out, 2 where the row is
    // near: those with an x filter are left to near_rows.
    template <int N3>
    __device__ __forceinline__ int bfl_type(V2 *out, int fl, const int (&dst)[N3], const int (&src)[N3], int yset, int zset, int x0,
                                            int y, int z) const {
        const int NY = k.NY, nb = 2*k.NYD6, r = z*k.NYD6 + y + 3;
        if (T.bfl_flag[fl*nb + r] != 1) return 0;
        const size_t N = (size_t)NX*NY*k.NZ;
        const float q = T.bfl_q[fl*nb + r];
        if (q > 0.5f) {   // (1/(2Q)) f_opposite + ((2Q-1)/(2Q)) f at the node
            const S *nd = fo + ((size_t)z*NY + y)*NX + x0;
            const float c0 = 1.f/(2.f*q), c1 = (2.f*q - 1.f)/(2.f*q);
#pragma unroll
            for (int m = 0; m < N3; m++) out[m] = V2(c0)*ld2g<S>(nd + src[m]*N, src[m]) + V2(c1)*ld2g<S>(nd + dst[m]*N, dst[m]);
        }
        if (q < 0.5f) {
            const int iy = k.bfl_mode ? r : y + 3;   // reference: Y weights at [j]
            out[0] = bfl_y_xi(src[0], yset, zset, x0, y, r, iy);
            return 2;
        }
        return q > 0.5f ? 1 : 0;
    }

    // What the lower wall sets at planes z = 0 and 1 of a node pair: bounce-back (z = 0) and BFL rows. It
    // depends on the old state only, so a piece that starts at the wall computes it before its first
    // target, while the ring fills (after the ring it cost 2.6 us per plane, on the critical
    // path of small grids). Indexed at run time: it lives in local memory.
    struct Wall {
        V2 v[2][8];        // 3, 7, 8 | 4, 9, 10 | 15 | 16
        V2 bounce[5];      // 5, 11, 12, 15, 16 at z = 0
        unsigned set[2];   // BFL types set at plane z
    };
    // Called by all collide threads; own: the thread's row is this tile's
    __device__ __forceinline__ void prepare_wall(unsigned char *smem, Wall &w, int z0, int z1, int x0, int row, int y0, bool own) const {
        const size_t N = (size_t)NX*k.NY*k.NZ;
        const int y = y0 + row;
        if (z0 == 0 && own) {
            const S *b = fo + ((size_t)y*NX + x0);
            w.bounce[0] = ld2g<S>(b + 6*N, 6);
            w.bounce[1] = ld2g<S>(b + 14*N, 14);
            w.bounce[2] = ld2g<S>(b + 13*N, 13);
            w.bounce[3] = ld2g<S>(b + 18*N, 18);
            w.bounce[4] = ld2g<S>(b + 17*N, 17);
        }
#pragma unroll 1
        for (int z = z0; z < z1; z++) {
            V2 *v = w.v[z];
            int t[4] = {0, 0, 0, 0};
            if (own) {
                t[0] = bfl_type<3>(v, 0, {3, 7, 8}, {4, 10, 9}, B_YB378, B_XIB378, x0, y, z);
                t[1] = bfl_type<3>(v + 3, 1, {4, 9, 10}, {3, 8, 7}, B_YB4910, B_XIB4910, x0, y, z);
                t[2] = bfl_type<1>(v + 6, 2, {15}, {18}, B_YB15, B_XIB15, x0, y, z);
                t[3] = bfl_type<1>(v + 7, 3, {16}, {17}, B_YB16, B_XIB16, x0, y, z);
            }
            w.set[z] = (t[0] ? 1u : 0u) | (t[1] ? 2u : 0u) | (t[2] ? 4u : 0u) | (t[3] ? 8u : 0u);
            if constexpr (TY >= 8) near_rows(smem, v, z, x0, row, y0, t[0] == 2, t[1] == 2);
            else near_row(v, z, x0, y, t[0] == 2, t[1] == 2);
        }
    }

    // The populations with an x axis of the thread's row at plane z, where the row is near: 7, 8 (near0: type 0) and 9,
    // 10 (near1: type 1) into v[1], v[2] and v[4], v[5]. A (row, type) takes 14 sums of 7 x 7 terms, one per
    // population and plane, each about 1 us of load latency. One after the other, by the row's threads.
    __device__ __forceinline__ void near_row(V2 *v, int z, int x0, int y, bool near0, bool near1) const {
        const int r = z*k.NYD6 + y + 3, iy = k.bfl_mode ? r : y + 3;   // reference: Y weights at [j]
#pragma unroll 1
        for (int i = 0; i < 4; i++) {
            const int type = i >> 1, m = i & 1;
            if (!(type ? near1 : near0)) continue;
            V2 g = V2(0.f);
#pragma unroll 1
            for (int c = 0; c < 7; c++)
                g = V2(bw(type ? B_XIB4910 : B_XIB378, c, r))*bfl_x_y((type ? 8 : 10) - m, c, (type ? B_XB49 : B_XB37) + m,
                                                                      type ? B_YB4910 : B_YB378, x0, y, r, iy) + g;
            v[3*type + 1 + m] = g;
        }
    }
    // The same for tiles of eight or sixteen rows: every row's threads take one sum of any near row at a time, exchanged
    // through shared memory, and a near row's own threads add its planes in their order. Per step of one
    // solve on the steep hill (alpha 0.73), against near_row: 64x32x48 FP32 28.9 us (34.1), FP16 29.8 (38.3);
    // 128x64x96 61.0 (66.7) and 55.5 (60.3); a burst of twelve on 64x32x48 170 ms (185). Tiles of four
    // rows, as many of them near: 256x128x192 220 us (206).
    __device__ __forceinline__ void near_rows(unsigned char *smem, V2 *v, int z, int x0, int row, int y0, bool near0, bool near1) const {
        volatile int *list = (volatile int *)(smem + LY::near_off) + z*(1 + 2*TY);   // number of entries, 2*row + type
        V2 *mids = (V2 *)(smem + LY::mids_off);                                      // [TY][PR]
        float *wz = (float *)(smem + LY::wz_off);                                    // [TY], the xi weight of each sum
        const int j = x0/2;
        if (j == 0 && near0) list[1 + atomicAdd((int *)list, 1)] = 2*row;
        if (j == 0 && near1) list[1 + atomicAdd((int *)list, 1)] = 2*row + 1;
        __syncwarp();
        bar_sync(BAR_COLLIDE, COLLIDE_THREADS);
        const int entries = list[0];
        if (entries == 0) {
            bar_sync(BAR_COLLIDE, COLLIDE_THREADS);   // every thread has read it before the next wall piece adds to it
            return;
        }
        int at[2] = {0, 0};
        for (int i = 0; i < entries; i++) {
            if (list[1 + i] == 2*row) at[0] = 14*i;
            if (list[1 + i] == 2*row + 1) at[1] = 14*i;
        }
        V2 g[2][2] = {{V2(0.f), V2(0.f)}, {V2(0.f), V2(0.f)}};
#pragma unroll 1
        for (int base = 0; base < 14*entries; base += TY) {
            if (base + row < 14*entries) {
                const int e = list[1 + (base + row)/14], s = (base + row) % 14, m = s >= 7 ? 1 : 0, type = e & 1, ye = y0 + (e >> 1);
                const int r = z*k.NYD6 + ye + 3, iy = k.bfl_mode ? r : ye + 3;   // reference: Y weights at [j]
                if (j == 0) wz[row] = bw(type ? B_XIB4910 : B_XIB378, s - 7*m, r);
                mids[row*PR + j] = bfl_x_y((type ? 8 : 10) - m, s - 7*m, (type ? B_XB49 : B_XB37) + m, type ? B_YB4910 : B_YB378, x0, ye, r, iy);
            }
            __syncwarp();
            bar_sync(BAR_COLLIDE, COLLIDE_THREADS);
#pragma unroll
            for (int type = 0; type < 2; type++)
                if (type ? near1 : near0)
#pragma unroll
                    for (int m = 0; m < 2; m++) {
                        const int first = at[type] + 7*m;
                        for (int s = max(base, first); s < min(base + TY, first + 7); s++)
                            g[type][m] = V2(wz[s - base])*mids[(s - base)*PR + j] + g[type][m];
                    }
            if (base + TY >= 14*entries && row == 0 && j == 0) list[0] = 0;   // for the next wall piece
            __syncwarp();
            bar_sync(BAR_COLLIDE, COLLIDE_THREADS);
        }
        if (near0) { v[1] = g[0][0]; v[2] = g[0][1]; }
        if (near1) { v[4] = g[1][0]; v[5] = g[1][1]; }
    }

    // Walls, BFL rows, collision and stores of the node pair (x0, x0 + 1) at row y, plane z, whose
    // streamed populations are in F (deviations for the deviation formats)
    // (WALL: z <= 1, the planes that the lower wall sets)
    template <bool WALL>
    __device__ __forceinline__ void finish(V2 (&F)[19], int x0, int y, int z, const Scal &sc, float &ub, V2 &mass, const Wall *wall) const {
        const int NY = k.NY;
        const size_t N = (size_t)NX*NY*k.NZ;
        // byte offsets fit 32 bits (roles_supported): a uniform base and a 32-bit offset per store
        // instead of a 64-bit address each (FP16 193 -> 182 us per step on 256x128x192)
        const unsigned node = (unsigned)((z*NY + y)*NX + x0), off = node*(unsigned)sizeof(S), moff = node*4u;
        const S *b = (const S *)((const char *)fo + off);
        if constexpr (Storage<S>::dev) {
#pragma unroll
            for (int q = 0; q < 19; q++) F[q] = F[q] + V2((float)dev_ref(q));
        }
        if constexpr (WALL) {
            if (z == 0) { F[5] = wall->bounce[0]; F[11] = wall->bounce[1]; F[12] = wall->bounce[2]; F[15] = wall->bounce[3]; F[16] = wall->bounce[4]; }
            const V2 *v = wall->v[z];
            const unsigned m = wall->set[z];
            if (m & 1u) { F[3] = v[0]; F[7] = v[1]; F[8] = v[2]; }
            if (m & 2u) { F[4] = v[3]; F[9] = v[4]; F[10] = v[5]; }
            if (m & 4u) F[15] = v[6];
            if (m & 8u) F[16] = v[7];
        }
        if (z == k.NZ - 1) {
            F[6] = ld2g<S>(b + 5*N, 5); F[13] = ld2g<S>(b + 12*N, 12); F[14] = ld2g<S>(b + 11*N, 11);
            F[17] = ld2g<S>(b + 16*N, 16); F[18] = ld2g<S>(b + 15*N, 15);
        }
        V2 rho, u1, v1, w1;
        collide_x2<LES>(F, sc.rho_mod, sc.f6, sc.f12, sc.tau, sc.lesC, rho, u1, v1, w1);
#pragma unroll
        for (int q = 0; q < 19; q++) st2<S>((S *)((char *)fnq[q] + off), F[q], q);
        if (macros_on) {
            *(float2 *)((char *)rho_out + moff) = rho.v; *(float2 *)((char *)u_out + moff) = u1.v;
            *(float2 *)((char *)v_out + moff) = v1.v; *(float2 *)((char *)w_out + moff) = w1.v;
        }
        // column partials in FP32, at most 16 terms (collide_piece)
        if (y == k.yplane) ub += (v1.v.x*T.dxf[x0] + v1.v.y*T.dxf[x0 + 1])*T.dzf[z];
        mass = mass + rho;   // a non-finite density makes the mass sum non-finite (checked once per piece)
    }

    // A collide warp's node pair and its place in the pipelines
    struct Pair {
        int w, i, row, x0, y;      // lane quarter, pair in the tile, row and columns
        int freed;                 // first ring plane not yet released
        unsigned seq0, tcount;     // ring sequence number of plane p0, target stages used
        uint32_t tl;
        bool own;                  // false: the previous tile's row
    };
    // Targets t0 .. t1 - 1 of a piece
    template <bool WALL>
    __device__ __forceinline__ void collide_targets(unsigned char *smem, const Piece &P, int t0, int t1, Pair &L, int lane, const Scal &sc,
                                                    float &ub, V2 &mass, bool &faulted, const Wall *wall) const {
#pragma unroll 1
        for (int t = t0; t < t1; t++, L.tcount++) {
            const int st = (int)(L.tcount % LY::NTS), base = window_base(t);
            const unsigned char *stage = smem + LY::target_off + st*LY::target_bytes;
            V2 F[19];
            __syncwarp();   // (rows of one warp may have parted at the walls, the ring loads are warp-wide)
            wait(smem, LY::B_TF + st, (L.tcount/LY::NTS) & 1u, faulted);
            const unsigned seq = L.seq0 + (unsigned)(base - P.p0), last = seq + 6;
            wait(smem, LY::B_RF + L.w*SLOTS + (int)(last % SLOTS), (last/SLOTS) & 1u, faulted);
            tmem_fence_after();
            xi_combine(L.tl, seq, (const float4 *)(stage + LY::w_off) + L.row*32, F, [&] {
                const S *q0 = (const S *)stage + L.row*NX;
                float o[4];
                F[0] = ld2v<S>(q0 + L.x0);
                x_filter(q0 + TY*NX, L.i % PR, 0, o[0], o[1]);
                x_filter(q0 + 2*TY*NX, L.i % PR, 1, o[2], o[3]);
                F[1] = V2(o[0], o[1]);
                F[2] = V2(o[2], o[3]);
            });
            tmem_fence_before();
            __syncwarp();
            // planes below the next target's window are free; so is the target stage
            const int next = t + 1 < P.tb ? window_base(t + 1) : P.p1 + 1;
            if (lane == 0) {
                mbar_arrive(bars(smem, LY::B_TE + st));
                for (int p = L.freed; p < next; p++)
                    mbar_arrive(bars(smem, LY::B_RE + L.w*SLOTS + (int)((L.seq0 + (unsigned)(p - P.p0)) % SLOTS)));
            }
            L.freed = next;
            if (L.own) finish<WALL>(F, L.x0, L.y, t, sc, ub, mass, wall);
        }
    }
    // All targets of a piece for collide warp `warp` (lane quarter warp % 4, row of the pair warp / 4);
    // seq0: ring sequence number of plane p0, tcount: target stages used before this piece. The wall
    // planes run in a loop of their own, so that the main one carries none of their state. The sums of the plane
    // velocity and the density are added in FP32 over FOLD targets, 16 with the two wall planes (the paired
    // kernel's segments have 16 or more), then in FP64 in the thread's word `sums` in shared memory: a segment may be the
    // whole column, 84 targets on 128x256x192. (In registers the FP64 sums cost 204 instead of 196 us there;
    // FP32 sums with their rounding errors beside them 206 to 226.)
    static constexpr int FOLD = 14;
    __device__ __forceinline__ void collide_piece(unsigned char *smem, const Piece &P, unsigned seq0, unsigned tcount, int warp, int lane,
                                                  uint32_t tl, const Scal &sc, double2 *sums, bool &faulted) const {
        float ub = 0.f;
        V2 mass = V2(0.f);
        auto fold = [&] {
            double2 s = *sums;
            s.x += (double)ub;
            s.y += (double)(mass.v.x + mass.v.y);
            *sums = s;
            ub = 0.f;
            mass = V2(0.f);
        };
        Pair L;
        L.w = warp & 3;
        L.i = 32*L.w + lane;
        L.row = 2*(L.i/PR) + (warp >> 2);
        L.x0 = 2*(L.i % PR);
        L.y = P.y0 + L.row;
        L.freed = P.p0;
        L.seq0 = seq0;
        L.tcount = tcount;
        L.tl = tl;
        L.own = L.row >= P.yskip;
        if (P.ta <= 1) {
            Wall wall;
            prepare_wall(smem, wall, P.ta, min(P.tb, 2), L.x0, L.row, P.y0, L.own);
            collide_targets<true>(smem, P, P.ta, min(P.tb, 2), L, lane, sc, ub, mass, faulted, &wall);
        }
#pragma unroll 1
        for (int t = max(P.ta, 2); t < P.tb; t += FOLD) {
            collide_targets<false>(smem, P, t, min(t + FOLD, P.tb), L, lane, sc, ub, mass, faulted, nullptr);
            fold();
        }
        if (P.tb <= 2) fold();   // a segment of wall planes only
        if (!isfinite(sums->y)) ctrl->nonfinite = 1u;
    }

    // ---- CTA set-up and end ----

    __device__ __forceinline__ Scal scalars() const {
        Scal sc;
        const double force = ctrl->force;
        sc.f6 = (float)(1.0/6*force*k.dt);
        sc.f12 = (float)(1.0/12*force*k.dt);
        sc.rho_mod = (float)ctrl->rho_modify;
        sc.tau = (float)k.tau;
        sc.lesC = (float)k.les_C;
        return sc;
    }
    __device__ static void init(unsigned char *smem, int tid) {
        if (tid < 32) {
            if (tid == 0) {
                uint64_t *b = (uint64_t *)(smem + LY::bar_off);
                for (int i = 0; i < LY::NFS; i++) { mbar_init(b + LY::B_FF + i, 1); mbar_init(b + LY::B_FE + i, FILTER_WARPS); }
                for (int i = 0; i < LY::NTS; i++) { mbar_init(b + LY::B_TF + i, 1); mbar_init(b + LY::B_TE + i, COLLIDE_WARPS); }
                for (int i = 0; i < 4*SLOTS; i++) { mbar_init(b + LY::B_RF + i, 2); mbar_init(b + LY::B_RE + i, 2); }
                *(volatile int *)(smem + LY::flag_off) = 0;
                for (int z = 0; z < 2; z++) ((volatile int *)(smem + LY::near_off))[z*(1 + 2*TY)] = 0;
                fence_mbar_init();
            }
            __syncwarp();
            tmem_alloc((uint32_t *)(smem + LY::flag_off + 8), 512);
            tmem_relinquish();
        }
        tmem_fence_before();
        __syncthreads();
        tmem_fence_after();
    }
    // The CTA's place in the work list, by the SM it runs on: neighbouring tiles on neighbouring SMs share
    // the halo rows they read at the same time (256x128x192, without dependent launches: FP32 181
    // -> 178, FP16 181 -> 171 us per step; with an arbitrary placement 230 and 275, and dependent
    // launches place CTAs as SMs become free). Any placement is valid: a CTA takes the seat of its
    // SM or the next free one. (Grids smaller than the GPU go by block number.) The claim runs beside the
    // CTA's set-up. Launches take the two sets of seats in turn; the last CTA of a launch empties its set,
    // before the launch after next, which takes that set again, can start (a launch starts once every CTA of
    // the one before is past its wait for the end of the one before that). So nothing in a launch's
    // arguments marks a seat as taken, and a captured pair of launches can be replayed.
    __device__ __forceinline__ void claim_seat(unsigned char *smem, int tid) const {
        if (tid != 32) return;   // not the warp that allocates tensor memory
        const unsigned n = gridDim.x;
        unsigned s = blockIdx.x;
        if (tc.seats && n <= (unsigned)MAX_SEATS) {
            unsigned sm;
            asm volatile("mov.u32 %0, %smid;" : "=r"(sm));
            unsigned *seats = ctrl_seats(ctrl, seat_set);
            s = sm < n ? sm : n - 1;
            for (unsigned i = 1; i < n && atomicExch(seats + s, 1u) != 0u; i++) s = s + 1 == n ? 0 : s + 1;
        }
        *(volatile int *)(smem + LY::flag_off + 4) = (int)s;
    }
    __device__ static uint32_t tmem_base(unsigned char *smem) { return *(volatile uint32_t *)(smem + LY::flag_off + 8); }
    // by the collide warps, after their last use of the ring; the filter warps arrive after their last
    // store (ring_done), so that none is under way even after a timed-out pipeline
    __device__ static void ring_done() {
        tmem_wait_st();
        tmem_fence_before();
        bar_arrive(BAR_RING_END, RING_THREADS);
    }
    __device__ static void ring_free(unsigned char *smem, int tid) {
        tmem_fence_before();
        bar_sync(BAR_RING_END, RING_THREADS);
        if (tid < 32) {
            tmem_fence_after();
            tmem_dealloc(tmem_base(smem), 512);
        }
    }

    __device__ __forceinline__ void run(unsigned char *smem, const CUtensorMap *tm) const {
        const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
        if (smem_u32(smem) & 127u) tm = nullptr;   // tensor copies need 128-byte aligned destinations
        claim_seat(smem, tid);
        init(smem, tid);
        const int seat = *(volatile int *)(smem + LY::flag_off + 4);
        grid_dependency_wait();   // nothing above touches global memory but the seats
        bool faulted = false;
        if (warp < COLLIDE_WARPS) {
            regs_inc<Regs<S>::collide>();
            const uint32_t tl = tmem_base(smem) + ((uint32_t)(32*(warp & 3)) << 16) + 256u*(uint32_t)(warp >> 2);
            double2 *sums = (double2 *)(smem + LY::sums_off) + tid;
            *sums = make_double2(0.0, 0.0);
            const Scal sc = scalars();
            unsigned seq = 0, tcount = 0;
            for_items(seat, [&](const Piece &P) {
                collide_piece(smem, P, seq, tcount, warp, lane, tl, sc, sums, faulted);
                seq += (unsigned)(P.p1 - P.p0 + 1);
                tcount += (unsigned)(P.tb - P.ta);
            });
            // the next step's CTAs may come now: triggered at the start, they took SMs one by one as
            // these became free, which scatters neighbouring tiles
            grid_dependency_trigger();
            ring_free(smem, tid);
            const bool last = end_of_step_ordered<COLLIDE_THREADS>(ctrl, k, tc.n, sums->x, sums->y, mass_on != 0, (unsigned)seat,
                                                                   gridDim.x, tid, [] { bar_sync(BAR_COLLIDE, COLLIDE_THREADS); });
            if (last && tid < MAX_SEATS) ctrl_seats(ctrl, seat_set)[tid] = 0u;   // (every CTA took its seat long ago)
        } else if (warp < FRONT_WARP) {
            if (warp < FILTER_WARP0 + 4) regs_dec<Regs<S>::rows>();
            else regs_dec<Regs<S>::quads>();
            const int w = warp - FILTER_WARP0;
            const uint32_t tl = tmem_base(smem) + ((uint32_t)(32*(w & 3)) << 16);
            unsigned seq = 0;
            Stage<LY::NFS> at;
            for_items(seat, [&](const Piece &P) { filter_planes(smem, P, at, seq, w, lane, tl, faulted); });
            ring_done();
        } else {
            regs_dec<Regs<S>::copies>();
            unsigned count = 0;
            if (warp == FRONT_WARP && lane == 0) {
                Stage<LY::NFS> at;
                for_items(seat, [&](const Piece &P) { produce_front(smem, P, at, count, faulted, tm); });
                drain(smem, LY::B_FF, LY::NFS, count);
            } else if (warp == TARGET_WARP && lane == 0) {
                Stage<LY::NTS> at;
                for_items(seat, [&](const Piece &P) { produce_targets(smem, P, at, count, faulted, tm); });
                drain(smem, LY::B_TF, LY::NTS, count);
            }
        }
    }
};

template <class S, bool LES, int NXC>
__global__ void __launch_bounds__(THREADS, 1)
step_roles_kernel(const __grid_constant__ RoleKernel<S, LES, NXC> K, const __grid_constant__ RoleTM T, int tm_on) {
    extern __shared__ __align__(128) unsigned char smem[];
    K.run(smem, tm_on ? T.m : nullptr);
}

// Batched form (serving): work items (solve, segment*ntiles + tile) of many solves of the same
// storage format and width; for each item the CTA copies the solve's descriptor into shared memory
// and takes the buffers from the solve's own step counter (a graph of identical launches advances
// every solve step after step).
template <class S, bool LES, int NXC>
struct RoleBatchDesc {
    CUtensorMap tm[2][5];   // tensor maps of buf[0], buf[1] (used when tm_on)
    RoleKernel<S, LES, NXC> K;
    S *buf[2];              // population buffers; the old one is buf[step & 1]
    int ntiles, nseg;
    int tm_on;
};

template <class S, bool LES, int NXC>
__global__ void __launch_bounds__(THREADS, 1)
step_roles_batch_kernel(const RoleBatchDesc<S, LES, NXC> *__restrict__ descs, const int2 *__restrict__ items, int nitems, int macros_on) {
    using KT = RoleKernel<S, LES, NXC>;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(16) unsigned char kbuf[sizeof(KT)];
    __shared__ unsigned long long step_s;
    KT &K = *(KT *)kbuf;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    KT::init(smem, tid);
    grid_dependency_wait();
    bool faulted = false;
    // the descriptor of item `it` into K, by the 18 active warps together
    auto load_item = [&](int it, int2 &w, const CUtensorMap *&tm) {
        w = items[it];
        bar_sync(BAR_ITEM, ACTIVE_THREADS);   // every role is done with the previous item
        const unsigned *src = (const unsigned *)&descs[w.x].K;
        for (int i = tid; i < (int)(sizeof(KT)/4); i += ACTIVE_THREADS) ((unsigned *)kbuf)[i] = src[i];
        if (tid == 0) step_s = *(volatile unsigned long long *)&descs[w.x].K.ctrl->step;
        bar_sync(BAR_ITEM, ACTIVE_THREADS);
        if (tid == 0) {
            const unsigned long long st = step_s;
            K.fo = descs[w.x].buf[st & 1ULL];
            K.fn = descs[w.x].buf[(st + 1) & 1ULL];
            const size_t N = (size_t)K.k.NX*K.k.NY*K.k.NZ;
            for (int q = 0; q < 19; q++) K.fnq[q] = K.fn + q*N;
            K.tc.n = st + 1;
            K.mass_on = K.k.mass_interval > 0 && ((st + 1) % (unsigned long long)K.k.mass_interval) == 0ULL;
            K.macros_on = macros_on;
        }
        bar_sync(BAR_ITEM, ACTIVE_THREADS);
        tm = descs[w.x].tm_on && !(smem_u32(smem) & 127u) ? descs[w.x].tm[step_s & 1ULL] : nullptr;
        const int nt = descs[w.x].ntiles, ns = descs[w.x].nseg, seg = w.y/nt;
        return K.make_piece(w.y - seg*nt, (int)((long long)seg*K.k.NZ/ns), (int)((long long)(seg + 1)*K.k.NZ/ns));
    };
    int2 w;
    const CUtensorMap *tm;
    if (warp < COLLIDE_WARPS) {
        regs_inc<Regs<S>::collide>();
        const uint32_t tl = KT::tmem_base(smem) + ((uint32_t)(32*(warp & 3)) << 16) + 256u*(uint32_t)(warp >> 2);
        unsigned seq = 0, tcount = 0;
        double2 *sums = (double2 *)(smem + KT::LY::sums_off) + tid;
        for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
            const typename KT::Piece P = load_item(it, w, tm);
            const auto sc = K.scalars();
            *sums = make_double2(0.0, 0.0);
            K.collide_piece(smem, P, seq, tcount, warp, lane, tl, sc, sums, faulted);
            seq += (unsigned)(P.p1 - P.p0 + 1);
            tcount += (unsigned)(P.tb - P.ta);
            end_of_step_ordered<COLLIDE_THREADS>(K.ctrl, K.k, K.tc.n, sums->x, sums->y, K.mass_on != 0, (unsigned)w.y,
                                                 (unsigned)(descs[w.x].ntiles*descs[w.x].nseg), tid,
                                                 [] { bar_sync(BAR_COLLIDE, COLLIDE_THREADS); });
        }
        grid_dependency_trigger();
        KT::ring_free(smem, tid);
    } else if (warp < FRONT_WARP) {
        if (warp < FILTER_WARP0 + 4) regs_dec<Regs<S>::rows>();
        else regs_dec<Regs<S>::quads>();
        const uint32_t tl = KT::tmem_base(smem) + ((uint32_t)(32*(warp & 3)) << 16);
        unsigned seq = 0;
        typename KT::template Stage<KT::LY::NFS> at;
        for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
            const typename KT::Piece P = load_item(it, w, tm);
            K.filter_planes(smem, P, at, seq, warp - FILTER_WARP0, lane, tl, faulted);
        }
        KT::ring_done();
    } else {
        regs_dec<Regs<S>::copies>();
        if (warp > TARGET_WARP) return;
        unsigned count = 0;
        typename KT::template Stage<KT::LY::NFS> fat;
        typename KT::template Stage<KT::LY::NTS> tat;
        for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
            const typename KT::Piece P = load_item(it, w, tm);
            if (lane == 0) {
                if (warp == FRONT_WARP) K.produce_front(smem, P, fat, count, faulted, tm);
                else K.produce_targets(smem, P, tat, count, faulted, tm);
            }
            __syncwarp();
        }
        if (lane == 0 && count) {
            if (warp == FRONT_WARP) K.drain(smem, KT::LY::B_FF, KT::LY::NFS, count);
            else K.drain(smem, KT::LY::B_TF, KT::LY::NTS, count);
        }
    }
}

template <class S, bool LES, int NXC>
struct RoleOps {
    using KT = RoleKernel<S, LES, NXC>;
    using D = RoleBatchDesc<S, LES, NXC>;
    static constexpr int smem = RLay<S, NXC>::smem_bytes;

    static cudaError_t launch(const StepLaunch &L) {
        KT K;
        K.fo = (const S *)L.fo;
        K.fn = (S *)L.fn;
        for (int q = 0; q < 19; q++) K.fnq[q] = K.fn + (size_t)q*L.k.NX*L.k.NY*L.k.NZ;
        K.T = *(const Tables<float> *)L.tables;
        K.k = L.k;
        K.tc = *(const TiledConst *)L.tiled;
        K.tc.n = L.n;
        K.ctrl = L.ctrl;
        K.rho_out = (float *)L.macros[0]; K.u_out = (float *)L.macros[1];
        K.v_out = (float *)L.macros[2]; K.w_out = (float *)L.macros[3];
        K.macros_on = L.macros_on; K.mass_on = L.mass;
        K.seat_set = L.seat_set;
        RoleTM T;
        std::memset((void *)&T, 0, sizeof(T));
        if (L.pmaps) std::memcpy((void *)T.m, L.pmaps, sizeof(T.m));
        return launch_dependent(step_roles_kernel<S, LES, NXC>, K.tc.grid, THREADS, smem, L.stream, K, T, (int)(L.pmaps != nullptr));
    }
    static size_t desc_bytes() { return sizeof(D); }
    static void fill(const Tables<float> &T, const StepConst &k, const TiledConst &tc, Ctrl *ctrl, void *const macros[4],
                     void *const buf[2], const RoleMaps &maps, int ntiles, int nseg, void *out) {
        D d;
        std::memset((void *)&d, 0, sizeof(d));
        d.K.T = T; d.K.k = k; d.K.tc = tc; d.K.ctrl = ctrl;
        d.K.rho_out = (float *)macros[0]; d.K.u_out = (float *)macros[1];
        d.K.v_out = (float *)macros[2]; d.K.w_out = (float *)macros[3];
        d.buf[0] = (S *)buf[0]; d.buf[1] = (S *)buf[1];
        d.ntiles = ntiles;
        d.nseg = nseg;
        d.tm_on = maps.ok && maps.buf[0] == buf[0] && maps.buf[1] == buf[1];
        if (d.tm_on) std::memcpy((void *)d.tm, (const void *)maps.m, sizeof(d.tm));
        std::memcpy(out, (const void *)&d, sizeof(d));
    }
    static cudaError_t launch_batch(const void *descs, const int2 *items, int nitems, int grid, int macros_on, cudaStream_t st) {
        return launch_dependent(step_roles_batch_kernel<S, LES, NXC>, grid, THREADS, smem, st, (const D *)descs, items, nitems, macros_on);
    }
    // on the current device; every solve does this at its set-up, before any launch or capture
    static cudaError_t prepare() {
        cudaError_t e = cudaFuncSetAttribute(step_roles_kernel<S, LES, NXC>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
        return cudaFuncSetAttribute(step_roles_batch_kernel<S, LES, NXC>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    }
};

// the operations of one storage format, for the dispatch of step_roles.cu
template <class S>
RoleTable role_table() {
    RoleTable t;
    auto one = [&](auto ops, int les, int w) {
        using O = decltype(ops);
        t.e[les][w] = RoleEntry{&O::launch, &O::desc_bytes, &O::fill, &O::launch_batch, &O::prepare, (size_t)O::smem};
    };
    one(RoleOps<S, false, 32>{}, 0, 0); one(RoleOps<S, false, 64>{}, 0, 1); one(RoleOps<S, false, 128>{}, 0, 2); one(RoleOps<S, false, 256>{}, 0, 3);
    one(RoleOps<S, true, 32>{}, 1, 0); one(RoleOps<S, true, 64>{}, 1, 1); one(RoleOps<S, true, 128>{}, 1, 2); one(RoleOps<S, true, 256>{}, 1, 3);
    return t;
}

}  // namespace
}  // namespace islbm
