// Chunk-marching step kernel: the separable interpolation on any grid in FP64 and FP32.
//
// Same step as stream_collide (C/evolution.h:358-684). It serves FP64 (the parity precision) and FP32 on
// every grid without a tiled layout (spanwise widths other than the tiled ones, streamwise counts
// that are no multiple of a tile's rows), where the gather kernel evaluates each departure point's
// 7 x 7 x 7 stencil by itself: about 2,500 multiply-adds and adds per node. Here the streamwise and
// spanwise filters are applied once per plane and node and the xi combination once per target,
// 252 multiply-adds per node, as the tiled kernels do:
//   * a CTA of four groups of threads owns a tile of W x H columns (one lane each of a group: at most 32 in
//     FP64, 64 in FP32) and marches upward through a wall-normal segment in chunks of CHUNK planes;
//   * phase A filters 7, 8, 9, 10 along one axis on the chunk's new planes into shared memory: FP64 in y, for the
//     tile's columns and three halo columns on each side; FP32 in x, for its rows and three halo rows on each
//     side; phase B filters them along the other axis, the other populations in y or x straight from
//     global memory (L1 / L2), and stores the 16 values of every column in a ring of CHUNK + 6 planes in
//     shared memory; phase C combines seven planes per target along xi, collides and stores. The four groups
//     take different planes (A, B) and targets (C) of a chunk, so a chunk costs two CTA barriers and no
//     other synchronisation;
//   * FP32 gives the gather kernel's bits: the same terms in the same order (see GATHER). Populations 3 and 4, whose xi
//     sums lie inside the y sum, cannot share a filtered plane; four targets share the loads of their windows;
//   * bounce-back (BFL) rows: the sums of the flagged rows are spread over the whole CTA before phase C.
//     The gather kernel's per-thread 343-point sums were the critical path on small grids.
//
// Bound: in FP64 the FP64 pipe (GB300 issues 2 FP64 lanes per clock and SM: about 430 operations per
// node take 4.3 ms on 256x128x192); in FP32 the latency of its loads at 16 warps per SM. Measured against the
// gather kernel, per step: FP64 256x128x192 (LES) 28.2 -> 5.50 ms, FP64 64x32x48 506 -> 112 us, FP32
// 187x91x131 (LES) 2,956 -> 272 us (8.2 GLUPS; 182 us with y and xi sums shared by all populations, which
// changed the last place of the results).
#include <algorithm>
#include <type_traits>
#include <cstring>

#include "collide.cuh"
#include "step_common.cuh"
#include "step_launch.hpp"
#include "step_chunk.hpp"

namespace islbm {

namespace {

// columns of a tile, one lane each, and the groups of that many lanes that share a CTA's planes and targets
constexpr int GROUPS = 4;
template <class C> __host__ __device__ constexpr int lanes() { return sizeof(C) == 4 ? 64 : 32; }
constexpr int CHUNK = 8, RING = CHUNK + 6;
// planes filtered between two barriers: a segment's first chunk takes RING, the others CHUNK. FP32 takes that
// one in two parts, which leaves more of an SM's memory to the L1 cache
template <class C> __host__ __device__ constexpr int batch() { return sizeof(C) == 4 ? CHUNK : RING; }

// A sum of products, term j = 0, 1, ... (compile-time in unrolled loops). FP32: the roundings that the gather
// kernel's unrolled sums are compiled to, w0 v0 + round(w1 v1), then one fused term after the other.
template <class C> struct Sum {
    C s = 0, w0, v0;
    __device__ __forceinline__ void add(int j, C w, C v) {
        if constexpr (sizeof(C) == 8) s += w*v;
        else if (j == 0) { w0 = w; v0 = v; }
        else if (j == 1) s = __fmaf_rn(w0, v0, __fmul_rn(w, v));
        else s = __fmaf_rn(w, v, s);
    }
};

// four values of one node (FP32: one 16-byte access, FP64: two)
template <class C> struct alignas(16) Quad { C a, b, c, d; };

template <class C> __host__ __device__ constexpr size_t ring_bytes() { return (size_t)RING*4*lanes<C>()*sizeof(Quad<C>); }
// FP32: the streamed populations 3 and 4 of a chunk's targets
template <class C> __host__ __device__ constexpr size_t f34_bytes() { return sizeof(C) == 4 ? (size_t)CHUNK*2*lanes<C>()*sizeof(C) : 0; }

__device__ __forceinline__ int wrap_near(int v, int n) {   // v in [-n, 2n)
    return v < 0 ? v + n : (v >= n ? v - n : v);
}
__device__ __forceinline__ int wrap_any(int v, int n) {
    v %= n;
    return v < 0 ? v + n : v;
}

template <class S, bool LES>
struct Chunk {
    using C = typename Storage<S>::C;
    static constexpr int P = lanes<C>(), NT = GROUPS*P;
    const S *fq[19];           // old populations, one array each: uniform bases for 32-bit byte offsets
    S *fnq[19];
    Tables<C> T;
    StepConst k;
    ChunkConst cc;
    Ctrl *ctrl;
    unsigned long long n;
    C *rho_out, *u_out, *v_out, *w_out;
    C ux0[7], ux2[7], uy0[7], uy2[7];   // FP32: the weights of every node
    int macros_on, mass_on;

    // Order of the sums. FP64 filters 7, 8, 9, 10 in y, then x, then xi, and every population with a
    // y and a xi axis in y first: the least work. FP32 (GATHER) adds the terms in the gather kernel's order
    // (x, y, xi; 3 and 4 xi, then y) and gives the same bits as that kernel. At nodes where a velocity component
    // is near zero another order moved it by up to 2.6e-3 of itself (2e-5 is a run's bound).
    static constexpr bool GATHER = sizeof(C) == 4;

    // value of population q at a byte offset (chunk_supported: 32 bits), by a plain load (grid_dependency_wait).
    // 64-bit addresses, one per load, were 40% of the kernel's instructions (FP32 187x91x131 224 us per step).
    __device__ __forceinline__ C val(int q, unsigned off) const { return to_c(*(const S *)((const char *)fq[q] + off)); }
    static constexpr unsigned EB = sizeof(S);

    // Lagrange weights. FP64 takes each node's own: they differ from the first node's by the rounding
    // of the node positions (about 1e-14), which the 1e-12 parity over a thousand steps would see. FP32
    // takes the first node's from constant memory (make_chunk_const: equal for all nodes in FP32)
    __device__ __forceinline__ C wx0(int a, int x) const { if constexpr (sizeof(C) == 8) return __ldg(T.wx0 + (size_t)a*k.NX + x); else return ux0[a]; }
    __device__ __forceinline__ C wx2(int a, int x) const { if constexpr (sizeof(C) == 8) return __ldg(T.wx2 + (size_t)a*k.NX + x); else return ux2[a]; }
    __device__ __forceinline__ C wy0(int b, int y) const { if constexpr (sizeof(C) == 8) return __ldg(T.wy0 + (size_t)b*k.NY + y); else return uy0[b]; }
    __device__ __forceinline__ C wy2(int b, int y) const { if constexpr (sizeof(C) == 8) return __ldg(T.wy2 + (size_t)b*k.NY + y); else return uy2[b]; }

    __device__ __forceinline__ int base(int t) const { return min(max(t - 3, 0), k.NZ - 7); }

    __device__ __forceinline__ int wrap_x(int v) const {   // v in [-3, NX + W + 2]
        const int NX = k.NX;
        if (NX < 8) return wrap_any(v, NX);
        v = v < 0 ? v + NX : v;
        v = v >= NX ? v - NX : v;
        return v >= NX ? v - NX : v;
    }

    // phase A, FP64: y filter of 7, 8, 9, 10 on planes p0 .. p0 + np - 1, columns x0 - 3 .. x0 + W + 2
    __device__ __forceinline__ void halo_quads(Quad<C> *qb, int p0, int np, int x0, int y0) const {
        const int WH = cc.W + 6, HW = cc.H*WH, NX = k.NX, NY = k.NY;
        for (int i = threadIdx.x; i < np*HW; i += NT) {
            const int pl = (int)__umulhi((unsigned)i, cc.inv_hw), r = i - pl*HW, yl = (int)__umulhi((unsigned)r, cc.inv_wh), xx = r - yl*WH;
            const int y = y0 + yl;
            if (y >= NY) continue;
            const unsigned b = (unsigned)((p0 + pl)*NY*NX + wrap_x(x0 + xx - 3));
            C s7 = 0, s8 = 0, s9 = 0, s10 = 0;
#pragma unroll
            for (int j = 0; j < 7; j++) {
                const unsigned o = (b + (unsigned)(wrap_near(y - 3 + j, NY)*NX))*EB;
                const C w0 = wy0(j, y), w2 = wy2(j, y);
                s7 += w0*val(7, o);
                s8 += w0*val(8, o);
                s9 += w2*val(9, o);
                s10 += w2*val(10, o);
            }
            qb[i] = Quad<C>{s7, s8, s9, s10};
        }
    }

    struct Col {
        int x, y, xl, yl;
        bool on, row;        // a column of the tile; phase A of FP32: a column of the grid
        unsigned ro, xo[7];  // byte offsets within a plane: the spanwise stencil's nodes (FP32: in a row, and the row's)
        unsigned yo[7];      // and the streamwise stencil's
    };
    // phase A, FP32: x filter of 7, 8, 9, 10 on planes p0 .. p0 + np - 1, rows y0 - 3 .. y0 + H + 2
    __device__ __forceinline__ void halo_rows(Quad<C> *qb, int p0, int np, int y0, const Col &L, int g) const {
        const int RH = cc.H + 6, NX = k.NX, NY = k.NY, per = P/cc.W;
        if (!L.row) return;
        for (int line = g*per + L.yl; line < np*RH; line += GROUPS*per) {
            const int pl = (int)__umulhi((unsigned)line, cc.inv_hw), y = y0 + line - pl*RH - 3;
            if (y > NY + 2) continue;
            const unsigned b = (unsigned)(((p0 + pl)*NY + wrap_near(y, NY))*NX)*EB;
            Sum<C> s7, s8, s9, s10;
#pragma unroll
            for (int a = 0; a < 7; a++) {
                const unsigned o = b + L.xo[a];
                s7.add(a, wx0(a, L.x), val(7, o));
                s8.add(a, wx2(a, L.x), val(8, o));
                s9.add(a, wx0(a, L.x), val(9, o));
                s10.add(a, wx2(a, L.x), val(10, o));
            }
            qb[line*cc.W + L.xl] = Quad<C>{s7.s, s8.s, s9.s, s10.s};
        }
    }

    // phase B: ring values of one column on one plane; ring order 3, 4, 5, 6 (FP32: 5, 6) |
    // 7, 8, 9, 10 | 11, 12, 13, 14 | 15, 16, 17, 18. qrow: the column's first quad of the plane
    __device__ __forceinline__ void filter(const Col &L, const Quad<C> *qrow, int p, Quad<C> *slot) const {
        const unsigned pl = (unsigned)(p*k.NY*k.NX)*EB;
        Sum<C> q[4];
        {
            Sum<C> g[2], h[4];
#pragma unroll
            for (int j = 0; j < 7; j++) {
                const unsigned o = pl + L.yo[j];
                const C w0 = wy0(j, L.y), w2 = wy2(j, L.y);
                if constexpr (GATHER) {
                    const Quad<C> v = qrow[j*cc.W];
                    q[0].add(j, w0, v.a);
                    q[1].add(j, w0, v.b);
                    q[2].add(j, w2, v.c);
                    q[3].add(j, w2, v.d);
                } else {
                    g[0].add(j, w0, val(3, o));
                    g[1].add(j, w2, val(4, o));
                }
                h[0].add(j, w0, val(15, o));
                h[1].add(j, w2, val(16, o));
                h[2].add(j, w0, val(17, o));
                h[3].add(j, w2, val(18, o));
            }
            slot[0*P] = Quad<C>{g[0].s, g[1].s, val(5, pl + L.yo[3]), val(6, pl + L.yo[3])};
            slot[3*P] = Quad<C>{h[0].s, h[1].s, h[2].s, h[3].s};
        }
        {
            Sum<C> h[4];
#pragma unroll
            for (int a = 0; a < 7; a++) {
                const unsigned o = pl + L.ro + L.xo[a];
                const C w0 = wx0(a, L.x), w2 = wx2(a, L.x);
                h[0].add(a, w0, val(11, o));
                h[1].add(a, w2, val(12, o));
                h[2].add(a, w0, val(13, o));
                h[3].add(a, w2, val(14, o));
                if constexpr (!GATHER) {
                    const Quad<C> v = qrow[a];
                    q[0].add(a, w0, v.a);
                    q[1].add(a, w2, v.b);
                    q[2].add(a, w0, v.c);
                    q[3].add(a, w2, v.d);
                }
            }
            slot[1*P] = Quad<C>{q[0].s, q[1].s, q[2].s, q[3].s};
            slot[2*P] = Quad<C>{h[0].s, h[1].s, h[2].s, h[3].s};
        }
    }

    // phase B, FP32: 3 and 4 of targets t0 .. t1 - 1 (at most CHUNK), xi inside y. A warp takes one of the two
    // populations for half of the targets; four targets read the 10 planes of their windows once.
    // f34[(t - t0)*2 + population][lane]
    __device__ __forceinline__ void y_of_xi(const Col &L, int t0, int t1, int g, C *f34) const {
        static_assert(GROUPS == 4 && CHUNK == 8, "two halves of four targets, two populations");
        const int pop = g & 1, first = t0 + 4*(g >> 1), last = min(first + 4, t1);
        const unsigned plane = (unsigned)(k.NY*k.NX)*EB;
        const S *f = pop ? fq[4] : fq[3];
        auto xiw = [&](int t, int c) -> C { return __ldg(T.wxi + ((size_t)t*k.NY + L.y)*64 + c*8 + pop); };
        auto at = [&](unsigned off) -> C { return to_c(*(const S *)((const char *)f + off)); };
        C *out = f34 + ((first - t0)*2 + pop)*P;
        if (last - first == 4 && base(last - 1) == base(first) + 3) {
            C w[4][7];
            Sum<C> o[4];
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int c = 0; c < 7; c++) w[i][c] = xiw(first + i, c);
#pragma unroll
            for (int b = 0; b < 7; b++) {
                const unsigned off = (unsigned)base(first)*plane + yo_at(L, b);
                const C wb = pop ? uy2[b] : uy0[b];
                C v[10];
#pragma unroll
                for (int p = 0; p < 10; p++) v[p] = at(off + (unsigned)p*plane);
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    Sum<C> in;
#pragma unroll
                    for (int c = 0; c < 7; c++) in.add(c, w[i][c], v[i + c]);
                    o[i].add(b, wb, in.s);
                }
            }
#pragma unroll
            for (int i = 0; i < 4; i++) out[2*i*P] = o[i].s;
            return;
        }
        for (int t = first; t < last; t++, out += 2*P) {   // windows held at a wall, or fewer targets
            Sum<C> o;
#pragma unroll 1
            for (int b = 0; b < 7; b++) {
                const unsigned off = (unsigned)base(t)*plane + yo_at(L, b);
                Sum<C> in;
#pragma unroll
                for (int c = 0; c < 7; c++) in.add(c, xiw(t, c), at(off + (unsigned)c*plane));
                o.add(b, pop ? uy2[b] : uy0[b], in.s);
            }
            *out = o.s;
        }
    }
    __device__ __forceinline__ unsigned yo_at(const Col &L, int b) const {
        return (unsigned)(wrap_near(L.y - 3 + b, k.NY)*k.NX + L.x)*EB;
    }

    // BFL rows: which sums a flagged row needs. Kinds 0..3 (with the halo columns): 7, 8, 9, 10 from
    // their opposites; kinds 4..7: 3, 4, 15, 16. The flag type of a kind and its source population
    // and weight sets (C/evolution.h:505-572).
    __device__ __forceinline__ static int kind_flag(int kd) { return kd < 2 ? 0 : kd < 4 ? 1 : kd - 4; }
    __device__ __forceinline__ static int kind_src(int kd) { return kd < 4 ? 10 - kd : kd == 4 ? 4 : kd == 5 ? 3 : kd == 6 ? 18 : 17; }
    __device__ __forceinline__ static int kind_xset(int kd) { return kd == 0 ? B_XB37 : kd == 1 ? B_XB38 : kd == 2 ? B_XB49 : B_XB410; }
    __device__ __forceinline__ static int kind_yset(int fl) { return fl == 0 ? B_YB378 : fl == 1 ? B_YB4910 : fl == 2 ? B_YB15 : B_YB16; }
    __device__ __forceinline__ static int kind_zset(int fl) { return fl == 0 ? B_XIB378 : fl == 1 ? B_XIB4910 : fl == 2 ? B_XIB15 : B_XIB16; }

    __device__ __forceinline__ C bw(int s, int a, int idx) const {
        const int nb = 2*k.NYD6;
        return idx < nb ? __ldg(T.bfl_w + ((size_t)s*7 + a)*nb + idx) : C(0);
    }

    // Sums of the flagged rows z = z0 .. z1 - 1 of the tile, bf[((z*H + yl)*8 + kind)*per + xx]. FP64: the (y, xi)
    // sums with the halo columns (per = W + 6); FP32: the whole sums (per = W). The flagged (row, kind)
    // pairs are listed first, so that all of them are summed in one pass of the CTA (row after row, their
    // load latencies add up).
    __device__ __forceinline__ void bfl_sums(C *bf, int z0, int z1, int x0, int y0) const {
        __shared__ int count;
        __shared__ unsigned short list[2*P*8];
        const int NX = k.NX, NY = k.NY, nb = 2*k.NYD6;
        if (threadIdx.x == 0) count = 0;
        __syncthreads();
        for (int i = z0*cc.H*8 + threadIdx.x; i < z1*cc.H*8; i += NT) {
            const int z = i/(8*cc.H), y = y0 + (i/8) % cc.H, fl = kind_flag(i & 7), r = z*k.NYD6 + y + 3;
            if (y < NY && T.bfl_flag[fl*nb + r] == 1 && T.bfl_q[fl*nb + r] < C(0.5)) list[atomicAdd(&count, 1)] = (unsigned short)i;
        }
        __syncthreads();
        const int per = GATHER ? cc.W : cc.W + 6, items = count*per;
        for (int i = threadIdx.x; i < items; i += NT) {
            const int m = i/per, xx = i - m*per, e = list[m], kd = e & 7, fl = kind_flag(kd), q = kind_src(kd);
            const int z = e/(8*cc.H), y = y0 + (e/8) % cc.H, r = z*k.NYD6 + y + 3;
            const int iy = k.bfl_mode ? r : y + 3;   // reference: Y weights at [j]
            if (GATHER && x0 + xx >= NX) continue;
            const unsigned b = (unsigned)(GATHER ? x0 + xx : wrap_x(x0 + xx - 3));
            const S *f = fq[q];
            C wy[7], sum = 0;
#pragma unroll
            for (int j = 0; j < 7; j++) wy[j] = bw(kind_yset(fl), j, iy);
            if (GATHER && kd < 4) {
                const int x = x0 + xx, ix = k.bfl_mode ? r : x + 3;
                C wx[7];
                unsigned xo[7];
#pragma unroll
                for (int a = 0; a < 7; a++) { wx[a] = bw(kind_xset(kd), a, ix); xo[a] = (unsigned)wrap_any(x - 3 + a, NX); }
#pragma unroll 1
                for (int c = 0; c < 7; c++) {
                    C mid = 0;
#pragma unroll
                    for (int j = 0; j < 7; j++) {
                        const unsigned row = (unsigned)((c*NY + wrap_near(y - 3 + j, NY))*NX);
                        C in = 0;
#pragma unroll
                        for (int a = 0; a < 7; a++) in += to_c(f[row + xo[a]])*wx[a];
                        mid += in*wy[j];
                    }
                    sum += mid*bw(kind_zset(fl), c, r);
                }
            } else {
#pragma unroll
                for (int c = 0; c < 7; c++) {
                    C in = 0;
#pragma unroll
                    for (int j = 0; j < 7; j++) in += to_c(f[b + (unsigned)((c*NY + wrap_near(y - 3 + j, NY))*NX)])*wy[j];
                    sum += in*bw(kind_zset(fl), c, r);
                }
            }
            bf[(size_t)e*per + xx] = sum;
        }
    }

    __device__ __forceinline__ void bfl_apply(C (&F)[19], const Col &L, int z, const C *bf) const {
        const int NX = k.NX, NY = k.NY, nb = 2*k.NYD6;
        const int r = z*k.NYD6 + L.y + 3;
        const int ix = k.bfl_mode ? r : L.x + 3;   // reference: X weights at [i]
        const unsigned nd = (unsigned)((z*NY + L.y)*NX + L.x)*EB;
        const int WH = GATHER ? cc.W : cc.W + 6;   // values of a kind
        const C *row = bf + (size_t)(z*cc.H + L.yl)*8*WH + L.xl;
        auto lin = [&](C q, int a, int b) -> C {   // (1/(2Q)) f_a + ((2Q-1)/(2Q)) f_b at the node
            return (C(1)/(C(2)*q))*val(a, nd) + ((C(2)*q - C(1))/(C(2)*q))*val(b, nd);
        };
        auto at = [&](int kd) -> C {
            return row[kd*WH + (GATHER ? 0 : 3)];
        };
        auto xf = [&](int kd, int set) -> C {
            if constexpr (GATHER) return at(kd);
            C s = 0;
#pragma unroll
            for (int a = 0; a < 7; a++) s += bw(set, a, ix)*row[kd*WH + a];
            return s;
        };
        if (T.bfl_flag[0*nb + r] == 1) {
            const C q = T.bfl_q[0*nb + r];
            if (q > C(0.5)) { F[3] = lin(q, 4, 3); F[7] = lin(q, 10, 7); F[8] = lin(q, 9, 8); }
            if (q < C(0.5)) { F[3] = at(4); F[7] = xf(0, B_XB37); F[8] = xf(1, B_XB38); }
        }
        if (T.bfl_flag[1*nb + r] == 1) {
            const C q = T.bfl_q[1*nb + r];
            if (q > C(0.5)) { F[4] = lin(q, 3, 4); F[9] = lin(q, 8, 9); F[10] = lin(q, 7, 10); }
            if (q < C(0.5)) { F[4] = at(5); F[9] = xf(2, B_XB49); F[10] = xf(3, B_XB410); }
        }
        if (T.bfl_flag[2*nb + r] == 1) {
            const C q = T.bfl_q[2*nb + r];
            if (q > C(0.5)) F[15] = lin(q, 18, 15);
            if (q < C(0.5)) F[15] = at(6);
        }
        if (T.bfl_flag[3*nb + r] == 1) {
            const C q = T.bfl_q[3*nb + r];
            if (q > C(0.5)) F[16] = lin(q, 17, 16);
            if (q < C(0.5)) F[16] = at(7);
        }
    }

    // phase C: target plane t of one column
    // (f34: FP32, the sums of y_of_xi for this target)
    __device__ __forceinline__ void target(const Col &L, const Quad<C> *ring, int t, const C *f34, const C *bf, C f6, C f12, C rho_mod,
                                           double &ub, double &mass) const {
        const int NX = k.NX, NY = k.NY;
        const int b = base(t);
        C F[19];
        {
            Sum<C> a[16];
            const Quad<C> *w = (const Quad<C> *)(T.wxi + ((size_t)t*NY + L.y)*64);
            int slot = b % RING;
#pragma unroll
            for (int c = 0; c < 7; c++) {
                const Quad<C> w0 = w[2*c], w1 = w[2*c + 1];   // xi 3, 4, 5, 6 | 15, 16, 17, 18
                const Quad<C> *v = ring + (size_t)slot*4*P;
                const Quad<C> v0 = v[0], v1 = v[P], v2 = v[2*P], v3 = v[3*P];
                if constexpr (!GATHER) { a[0].add(c, w0.a, v0.a); a[1].add(c, w0.b, v0.b); }
                a[2].add(c, w0.c, v0.c); a[3].add(c, w0.d, v0.d);
                const C m7[4] = {w0.a, w0.a, w0.b, w0.b}, f7[4] = {v1.a, v1.b, v1.c, v1.d};
#pragma unroll
                for (int m = 0; m < 4; m++) {   // (the gather kernel's loop over these is not unrolled)
                    if constexpr (GATHER) a[4 + m].s = __fmaf_rn(m7[m], f7[m], a[4 + m].s);
                    else a[4 + m].add(c, m7[m], f7[m]);
                }
                a[8].add(c, w0.c, v2.a); a[9].add(c, w0.c, v2.b); a[10].add(c, w0.d, v2.c); a[11].add(c, w0.d, v2.d);
                a[12].add(c, w1.a, v3.a); a[13].add(c, w1.b, v3.b); a[14].add(c, w1.c, v3.c); a[15].add(c, w1.d, v3.d);
                slot = slot == RING - 1 ? 0 : slot + 1;
            }
#pragma unroll
            for (int j = 0; j < 16; j++) F[3 + j] = a[j].s;
            if constexpr (GATHER) { F[3] = f34[0]; F[4] = f34[P]; }
        }
        const unsigned node = (unsigned)((t*NY + L.y)*NX + L.x), nd = node*EB;
        {
            const unsigned row = (unsigned)(t*NY*NX)*EB + L.ro;
            Sum<C> s1, s2;
#pragma unroll
            for (int a = 0; a < 7; a++) { s1.add(a, wx0(a, L.x), val(1, row + L.xo[a])); s2.add(a, wx2(a, L.x), val(2, row + L.xo[a])); }
            F[1] = s1.s; F[2] = s2.s;
            F[0] = val(0, nd);
        }
        auto opp = [&](int q) -> C { return val(q, nd); };
        if (t == 0) { F[5] = opp(6); F[11] = opp(14); F[12] = opp(13); F[15] = opp(18); F[16] = opp(17); }
        if (t == k.NZ - 1) { F[6] = opp(5); F[13] = opp(12); F[14] = opp(11); F[17] = opp(16); F[18] = opp(15); }
        if (t <= 1) bfl_apply(F, L, t, bf);
        C rho, u1, v1, w1;
        if constexpr (sizeof(C) == 4) collide_node<C, LES>(F, rho_mod, f6, f12, (C)k.tau, (C)k.les_C, rho, u1, v1, w1);
        else collide<LES>(F, rho_mod, f6, f12, k.tau, k.les_C, rho, u1, v1, w1);
#pragma unroll
        for (int q = 0; q < 19; q++) store_f<S>((S *)((char *)fnq[q] + nd), 0, q, F[q]);
        if (macros_on) { rho_out[node] = rho; u_out[node] = u1; v_out[node] = v1; w_out[node] = w1; }
        if (L.y == k.yplane) ub += (double)v1*T.dxv[L.x]*T.dzv[t];
        if (mass_on) mass += (double)rho;
        if (!(rho == rho)) ctrl->nonfinite = 1u;
    }

    __device__ __forceinline__ void run(unsigned char *smem) const {
        Quad<C> *ring = (Quad<C> *)smem;
        C *f34 = (C *)(smem + ring_bytes<C>());
        Quad<C> *qb = (Quad<C> *)(smem + ring_bytes<C>() + f34_bytes<C>());
        const int tid = threadIdx.x, c = tid % P, g = tid/P;
        const int NX = k.NX, NY = k.NY, NZ = k.NZ;
        double ub = 0.0, mass = 0.0;
        const double force = ctrl->force;
        const C f6 = (C)(1.0/6*force*k.dt), f12 = (C)(1.0/12*force*k.dt), rho_mod = (C)ctrl->rho_modify;
        const int ntiles = cc.tiles_x*cc.tiles_y;
        for (int item = blockIdx.x; item < ntiles*cc.segs; item += gridDim.x) {
            const int seg = item/ntiles, tile = item - seg*ntiles;
            const int ty = tile/cc.tiles_x, x0 = (tile - ty*cc.tiles_x)*cc.W, y0 = ty*cc.H;
            const int ta = (int)((long long)seg*NZ/cc.segs), tb = (int)((long long)(seg + 1)*NZ/cc.segs);
            Col L;
            L.yl = c/cc.W; L.xl = c - L.yl*cc.W;
            L.x = x0 + L.xl; L.y = y0 + L.yl;
            L.on = L.yl < cc.H && L.x < NX && L.y < NY;
            L.row = L.yl < P/cc.W && L.x < NX;
            const unsigned row = (unsigned)(L.y*NX)*EB;
            L.ro = GATHER ? row : 0u;
            if (GATHER ? L.row : L.on) {
#pragma unroll
                for (int a = 0; a < 7; a++) {
                    L.xo[a] = (unsigned)wrap_any(L.x - 3 + a, NX)*EB + (GATHER ? 0u : row);
                    L.yo[a] = (unsigned)(wrap_near(L.y - 3 + a, NY)*NX + L.x)*EB;
                }
            }
            int np = base(ta);   // next plane to filter
            for (int t0 = ta; t0 < tb; t0 += CHUNK) {
                const int t1 = min(t0 + CHUNK, tb);
                const int pend = base(t1 - 1) + 7;
                // planes np .. pb - 1: quads, then ring values
                auto planes = [&](int pb) {
                    if constexpr (GATHER) halo_rows(qb, np, pb - np, y0, L, g);
                    else halo_quads(qb, np, pb - np, x0, y0);
                    __syncthreads();   // quads complete; every thread is done with the previous chunk's targets
                    if (L.on)
                        for (int p = np + g; p < pb; p += GROUPS)
                            filter(L, qb + (GATHER ? ((p - np)*(cc.H + 6) + L.yl)*cc.W : ((p - np)*cc.H + L.yl)*(cc.W + 6)) + L.xl, p,
                                   ring + (size_t)(p % RING)*4*P + c);
                    np = pb;
                };
                if constexpr (GATHER)
                    while (pend - np > batch<C>()) {
                        planes(np + batch<C>());
                        __syncthreads();   // quads free
                    }
                planes(pend);
                if constexpr (GATHER) { if (L.on) y_of_xi(L, t0, t1, g, f34 + c); }
                __syncthreads();   // ring complete, quads free
                if (t0 <= 1) {
                    bfl_sums((C *)qb, t0, min(t1, 2), x0, y0);
                    __syncthreads();
                }
                if (L.on)
                    for (int t = t0 + g; t < t1; t += GROUPS)
                        target(L, ring + c, t, f34 + (t - t0)*2*P + c, (const C *)qb, f6, f12, rho_mod, ub, mass);
                if (t0 <= 1) __syncthreads();   // the sums are read before the next chunk's quads replace them
            }
        }
        end_of_step_ordered<NT>(ctrl, k, n, ub, mass, mass_on != 0, blockIdx.x, gridDim.x, tid, [] { __syncthreads(); });
    }
};

// CTAs per SM: shared memory (ring + quads) allows 3 in FP64 (about 71 KB) and 2 in FP32 (81 KB at 16x4);
// 168 registers per thread in FP64 and 128 in FP32
template <class S> constexpr int min_ctas() { return sizeof(typename Storage<S>::C) == 8 ? 3 : 2; }

template <class S, bool LES>
__global__ void __launch_bounds__(Chunk<S, LES>::NT, min_ctas<S>()) step_chunk_kernel(const __grid_constant__ Chunk<S, LES> K) {
    extern __shared__ __align__(128) unsigned char smem[];
    // the trigger comes after the wait: at most two steps are resident at a time
    grid_dependency_wait();
    grid_dependency_trigger();
    K.run(smem);
}

template <class C> size_t smem_for(int W, int H) {
    const bool rows = sizeof(C) == 4;   // halo rows (FP32) or halo columns
    const size_t quads = (size_t)batch<C>()*(rows ? (H + 6)*W : H*(W + 6))*sizeof(Quad<C>);
    const size_t sums = (size_t)2*H*8*(rows ? W : W + 6)*sizeof(C);
    return ring_bytes<C>() + f34_bytes<C>() + std::max(quads, sums);
}

template <class S, bool LES>
cudaError_t prepare_t(size_t smem, int *ctas) {
    cudaError_t e = cudaFuncSetAttribute(step_chunk_kernel<S, LES>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctas, step_chunk_kernel<S, LES>, Chunk<S, LES>::NT, smem);
}

template <class S, bool LES>
cudaError_t launch_t(const StepLaunch &L) {
    using C = typename Storage<S>::C;
    Chunk<S, LES> K;
    const size_t N = (size_t)L.k.NX*L.k.NY*L.k.NZ;
    for (int q = 0; q < 19; q++) { K.fq[q] = (const S *)L.fo + q*N; K.fnq[q] = (S *)L.fn + q*N; }
    K.T = *(const Tables<C> *)L.tables;
    K.k = L.k;
    K.cc = *(const ChunkConst *)L.chunk;
    K.ctrl = L.ctrl;
    K.n = L.n;
    K.rho_out = (C *)L.macros[0]; K.u_out = (C *)L.macros[1]; K.v_out = (C *)L.macros[2]; K.w_out = (C *)L.macros[3];
    for (int a = 0; a < 7; a++) {
        K.ux0[a] = (C)K.cc.wx0[a]; K.ux2[a] = (C)K.cc.wx2[a];
        K.uy0[a] = (C)K.cc.wy0[a]; K.uy2[a] = (C)K.cc.wy2[a];
    }
    K.macros_on = L.macros_on; K.mass_on = L.mass;
    return launch_dependent(step_chunk_kernel<S, LES>, K.cc.grid, Chunk<S, LES>::NT, K.cc.smem_bytes, L.stream, K);
}

template <class F>
cudaError_t by_kernel(int precision, bool les, F &&f) {
    if (precision == ISLBM_FP64) return les ? f((double *)nullptr, std::true_type{}) : f((double *)nullptr, std::false_type{});
    return les ? f((float *)nullptr, std::true_type{}) : f((float *)nullptr, std::false_type{});
}

}  // namespace

bool chunk_supported(const StepConst &k, int precision) {
    // 16-bit storage keeps the gather kernel's order of summation: each changed rounding of a stored value
    // is a visible change there
    if (precision != ISLBM_FP64 && precision != ISLBM_FP32) return false;
    const double elem = precision == ISLBM_FP64 ? 8 : 4;
    return (double)k.NX*k.NY*k.NZ*elem < 4294967296.0;
}

cudaError_t make_chunk_const(const StepConst &k, int precision, bool les, const double *wx0, const double *wx2,
                             const double *wy0, const double *wy2, int num_sms, ChunkConst *out) {
    ChunkConst cc;
    std::memset((void *)&cc, 0, sizeof(cc));
    for (int a = 0; a < 7; a++) { cc.wx0[a] = wx0[a]; cc.wx2[a] = wx2[a]; cc.wy0[a] = wy0[a]; cc.wy2[a] = wy2[a]; }
    const bool rows = precision != ISLBM_FP64;   // phase A takes halo rows (FP32) or halo columns
    const int P = rows ? lanes<float>() : lanes<double>();
    // wall-normal segments: rounds of items x (targets per segment + the ramp of 6 planes, whose
    // filters cost a quarter of a whole plane in FP64 and about half in FP32), down to one target
    // where a grid has few tiles
    const double ramp = precision == ISLBM_FP64 ? 1.5 : 3.0;
    auto makespan = [&](int tiles, int slots, int &segs) {
        double best = 1e300;
        for (int z = 1; z <= k.NZ; z++) {
            const long long items = (long long)tiles*z;
            const double rounds = (double)((items + slots - 1)/slots);
            const double cost = rounds*((double)((k.NZ + z - 1)/z) + ramp);
            if (cost < best - 1e-9) { best = cost; segs = z; }
        }
        return best;
    };
    // tile shape: a split of a row into equal parts of at most P columns, H rows of it. FP64: the fewest warps
    // per node; a part costs 32 lanes in phases B and C (about 0.95 of the work) and its halo columns
    // in phase A. FP32: the shortest makespan; a plane of a tile costs 1 + 0.0038 per halo-row value + 0.089
    // per row (the more rows, the shorter the runs of addresses): 187x91x131 in one round of 304 CTAs
    // 16x4 262 us per step, 12x5 272, 31x2 283, 8x8 285, and 13x4, which takes a second round, 350
    double best = 1e300;
    for (int parts = (k.NX + P - 1)/P; parts <= k.NX; parts++) {
        const int W = (k.NX + parts - 1)/parts, tx = (k.NX + W - 1)/W;
        const int H = std::min(P/W, k.NY), ty = (k.NY + H - 1)/H;
        double cost = (double)tx*ty*(0.95*P + 0.05*H*(W + 6));
        if (rows) {
            const int fit = (int)(228*1024/(smem_for<float>(W, H) + 4096));
            int z;
            cost = makespan(tx*ty, std::max(1, std::min(fit, min_ctas<float>()))*num_sms, z)*(1.0 + 0.0038*(H + 6)*W + 0.089*H);
        }
        if (cost < best*(1.0 - 1e-9)) { best = cost; cc.W = W; cc.H = H; cc.tiles_x = tx; cc.tiles_y = ty; }
        if (W <= 4) break;
    }
    const unsigned per_plane = (unsigned)(rows ? cc.H + 6 : cc.H*(cc.W + 6));
    cc.inv_hw = (unsigned)((0x100000000ULL + per_plane - 1)/per_plane);
    cc.inv_wh = (unsigned)((0x100000000ULL + cc.W + 5)/(cc.W + 6));
    cc.smem_bytes = precision == ISLBM_FP64 ? smem_for<double>(cc.W, cc.H) : smem_for<float>(cc.W, cc.H);
    int ctas = 0;
    cudaError_t e = by_kernel(precision, les, [&](auto *s, auto l) {
        using S = std::remove_pointer_t<decltype(s)>;
        return prepare_t<S, decltype(l)::value>(cc.smem_bytes, &ctas);
    });
    if (e != cudaSuccess) return e;
    if (ctas < 1) return cudaErrorInvalidConfiguration;
    const int tiles = cc.tiles_x*cc.tiles_y, slots = ctas*num_sms;
    makespan(tiles, slots, cc.segs);
    cc.grid = (int)std::min<long long>((long long)tiles*cc.segs, slots);
    *out = cc;
    return cudaSuccess;
}

cudaError_t launch_step_chunk(const StepLaunch &L) {
    return by_kernel(L.precision, L.les, [&](auto *s, auto l) {
        using S = std::remove_pointer_t<decltype(s)>;
        return launch_t<S, decltype(l)::value>(L);
    });
}

}  // namespace islbm
