// Host side of the role-specialised paired kernel (step_roles.cuh): dispatch by storage format, width
// and closure, column split, tensor maps.
#include <algorithm>
#include <cstdlib>
#include <cstring>

#include "step_roles.hpp"

namespace islbm {

namespace {

const RoleEntry &entry(int precision, int NX, bool les) {
    const RoleTable &t = precision == ISLBM_FP32 ? roles_fp32() : precision == ISLBM_FP16_DEV ? roles_fp16() : roles_bf16();
    return t.e[les ? 1 : 0][NX == 32 ? 0 : NX == 64 ? 1 : NX == 128 ? 2 : 3];
}

// A segment costs about this many targets more than its targets (the planes that fill the ring are
// filtered faster than targets are collided): from the busy times of SMs with one segment of 84
// targets and with two or three of 24 (407, 243 and 362 thousand cycles)
constexpr double RAMP = 2.0;

// Column split for `tiles` tiles on `slots` SMs, by the estimated makespan (a segment costs its targets
// + RAMP): either every column in zsegs equal segments, taken round by round, or zmain long
// segments per column, one per SM, and the rest of the columns on the SMs that are left.
void split_columns(int tiles, int slots, int NZ, TiledConst &tc) {
    tc.zmain = 0; tc.zlen = 0; tc.zsegs = 1;
    double best = 1e300;
    for (int z = 1; z <= NZ; z++) {
        const double rounds = (double)(((long long)tiles*z + slots - 1)/slots);
        const double cost = rounds*((double)((NZ + z - 1)/z) + RAMP);
        if (cost < best - 1e-9) { best = cost; tc.zsegs = z; }
    }
    const int m = slots/tiles, left = slots - m*tiles;
    if (m < 1 || left < 1) return;
    for (int zr = 1; zr <= 8; zr++)
        for (int len = 1; m*len < NZ; len++) {
            const int rest = NZ - m*len;
            if (rest < zr) continue;
            const double rounds = (double)(((long long)tiles*zr + left - 1)/left);
            const double cost = std::max((double)len + RAMP, rounds*((double)((rest + zr - 1)/zr) + RAMP));
            if (cost < best - 1e-9) { best = cost; tc.zmain = m; tc.zlen = len; tc.zsegs = zr; }
        }
}

}  // namespace

bool roles_supported(const StepConst &k, int precision) {
    if (precision == ISLBM_FP64) return false;
    if (k.NX != 32 && k.NX != 64 && k.NX != 128 && k.NX != 256) return false;
    // byte offsets into a population or field array are 32-bit in the kernel
    return k.NY >= 512/k.NX + 6 && k.NZ >= 8 && (double)k.NX*k.NY*k.NZ*4.0 < 4294967296.0;
}

cudaError_t make_roles_const(const StepConst &k, int precision, bool les, const double *wx0, const double *wx2,
                             const double *wy0, const double *wy2, int num_sms, TiledConst *out) {
    TiledConst tc;
    if (fill_pair_weights(wx0, wx2, wy0, wy2, &tc) != 0) return cudaErrorInvalidValue;
    tc.TY = 512/k.NX;
    const int tiles = (k.NY + tc.TY - 1)/tc.TY;
    split_columns(tiles, num_sms, k.NZ, tc);
    if (const char *e = std::getenv("ISLBM_TILED_ZSEGS")) {   // tuning override: equal segments
        const int z = std::atoi(e);
        if (z >= 1 && z <= k.NZ/8) { tc.zmain = 0; tc.zlen = 0; tc.zsegs = z; }
    }
    const long long items = (long long)tiles*(tc.zmain + tc.zsegs);
    tc.grid = tc.zmain ? num_sms : (int)std::min<long long>(items, num_sms);
    tc.seats = tc.grid == num_sms;
    *out = tc;
    const RoleEntry &e = entry(precision, k.NX, les);
    out->smem_bytes = e.smem;
    return e.prepare();
}

int roles_segments(int tiles, int slots, int NZ) {
    TiledConst tc;
    split_columns(tiles, slots, NZ, tc);
    return tc.zmain ? std::max(1, NZ/std::max(1, tc.zlen)) : tc.zsegs;
}

bool make_role_maps(const StepConst &k, int elem_bytes, void *const buf[2], RoleMaps *out) {
    out->ok = false;
    if ((elem_bytes != 4 && elem_bytes != 2) || !roles_supported(k, elem_bytes == 4 ? ISLBM_FP32 : ISLBM_FP16_DEV)) return false;
    const cuuint32_t TY = (cuuint32_t)(512/k.NX), NX = (cuuint32_t)k.NX;
    // box shapes: halo rows x 2 and 4 populations, tile rows x 2, 4 and 3 populations
    const cuuint32_t boxes[5][4] = {{NX, TY + 6, 1, 2}, {NX, TY + 6, 1, 4}, {NX, TY, 1, 2}, {NX, TY, 1, 4}, {NX, TY, 1, 3}};
    for (int b = 0; b < 2; b++)
        for (int j = 0; j < 5; j++)
            if (!encode_population_map(&out->m[b][j], k, elem_bytes, buf[b], boxes[j])) return false;
    out->buf[0] = buf[0];
    out->buf[1] = buf[1];
    out->ok = true;
    return true;
}

cudaError_t launch_step_roles(const StepLaunch &L) {
    return entry(L.precision, L.k.NX, L.les).launch(L);
}
size_t roles_batch_desc_bytes(int precision, int NX, bool les) {
    return entry(precision, NX, les).desc_bytes();
}
void fill_roles_batch_desc(int precision, int NX, bool les, const Tables<float> &T, const StepConst &k, const TiledConst &tc,
                           Ctrl *ctrl, void *const macros[4], void *const buf[2], const RoleMaps &maps, int ntiles, int nseg, void *out) {
    entry(precision, NX, les).fill(T, k, tc, ctrl, macros, buf, maps, ntiles, nseg, out);
}
cudaError_t launch_step_roles_batch(int precision, int NX, bool les, const void *descs, const int2 *items, int nitems, int grid,
                                    int macros_on, cudaStream_t stream) {
    return entry(precision, NX, les).launch_batch(descs, items, nitems, grid, macros_on, stream);
}

}  // namespace islbm
