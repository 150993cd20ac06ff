// k_raycast.cu -- predicted vertex / normal maps by ray marching the TSDF.
//
// Reference: raycastKernel (project/src/raycast.cu:44-145) with intersectBBox (:7-27) and
// computeGradient (:29-42), called once per pyramid level at the previous frame's pose
// (project/src/kinect_fusion.cpp:137-144).  The reference samples a cudaArray through the
// texture unit; here the distance array stays in linear HBM (x fastest), so fusion can stream
// it, and the march does its own trilinear interpolation with the reference's texel mapping
// (uvw * n - 0.5, clamp).  The march takes the reference's samples in the reference's order,
// with one difference in arithmetic: the reference forms each position by adding the step to
// the last one (t <- t + inc, project/src/raycast.cu:78), so float rounding drifts along a ray
// (up to ~1e-4 m over a grazing ray of a thousand small steps, which moves its hit by up to a
// millimetre); here sample k of a phase is at base + k * inc with a single rounding, where base
// is the near distance, the sample that left large steps, or t - mu after a back-off.  That is
// the FP64 march's position to within a rounding, and any sample's position is known without
// the ones before it.  Four things make the march fast:
//   - Depth ranges: the bricks that can end large steps, projected into 16 x 16-pixel tiles, tell
//     each ray the first and the last depth at which a sample can matter; it marches between them.
//   - Skipping: a sample whose eight taps lie in cells (32^3 super-bricks, then 8^3 bricks)
//     whose distance lower bound proves it cannot change the march (>= 0.991 during large
//     steps, >= 0.001 during small steps) is not evaluated, nor is any later sample in the
//     same cell; the march jumps to the first sample index past the cell.  A skip that starts
//     in a skippable super-brick continues through up to three more skippable super-bricks
//     along the ray (a run; longer runs let one lane hold its warp too long).  Rays that pass
//     within mu of a surface without crossing it keep 0.1 mu steps to the far plane (the
//     reference never returns to large steps); super-bricks let them cross free space 94 steps
//     at a time.
//   - Load balance: each warp pulls 8 x 4-ray tiles from an atomic counter, and a lane marches
//     at most 40 iterations (64 in steps of many sessions); longer rays are queued with their
//     exact march state.
//   - Long rays: a second kernel marches each queued ray with a whole warp, 32 consecutive
//     samples per round (64 after a round in which nothing changed), taking the first sample
//     (in order) that changes the state.
#include <algorithm>
#include <cmath>

#include "kf_host.h"

namespace kf {

constexpr int kMaxMarchSamples = 1 << 16;
// loop iterations a lane marches before queueing the ray: a short budget keeps the tail of a
// single session's frame short; steps of many sessions hand off fewer rays with a longer one.
// Measured, us: a frame of a 640x480 stream in 512^3 f32 193 with a budget of 24, 189 with 40, 199 with
// 64; 24 sessions of f16+u16 2,260 with 40, 2,243 with 64, 2,270 with 96.  The kernel's two forms go with
// the same line: 3 blocks per SM 189 and 2,405, 4 blocks 193 and 2,246 (320x240 in 128^3 118 and 129).
constexpr int kSerialBudgetSingle = 40;
constexpr int kSerialBudgetMany = 64;
constexpr int kManyRayTiles = 25000;   // more ray tiles than this in a step: kSerialBudgetMany
// skippable super-bricks one skip may cross.  Where no depth range starts a ray, free space is crossed by
// skips alone, and 4 cut the raycast's thread instructions by a third (32 sessions +8 %).  With the
// ranges, us: the stream's frame 189 at 1 and 4, 192 at 8 and 16; the 24 sessions 2,249, 2,243, 2,255
// and 2,261.
constexpr int kRunCells = 4;

bool many_ray_tiles(int ray_tiles) { return ray_tiles > kManyRayTiles; }
int serial_budget_many() { return kSerialBudgetMany; }
int serial_budget(int ray_tiles) { return many_ray_tiles(ray_tiles) ? kSerialBudgetMany : kSerialBudgetSingle; }

struct RayGeo {
    F3 o, dir;
    float sc, off;                            // texel coordinate = (o + dir t) * sc + off
    float tox, toy, toz, tdx, tdy, tdz;       // the same as an affine function of t
    float itdx, itdy, itdz;
};

// ---- depth ranges ----
//
// Most of a ray's samples lie in free space before its surface.  The bricks whose bound is below
// the large steps' threshold (a few percent of a volume) are projected into the level-0 image, and
// each kRangeTile^2-pixel tile keeps the nearest and the farthest camera depth at which a ray
// through it can have a sample in one of them.  Samples before the near depth or past the far one
// cannot change the march, in large steps or small ones (the small steps' threshold is lower), so
// a ray starts at the first sample index at or past the near depth and ends at the far depth: the
// same samples decide as before.  A ray's parameter t is its camera depth, and pixel (i, j) of
// level l passes through the point ((i + 1) 2^l - .5, (j + 1) 2^l - .5) of the level-0 image.
//
// What it measured: one 640x480 session in 512^3 f32, raycast kernel 94 -> 66 us and long rays 36 ->
// 31 us for a range launch of 5 to 9 us, a frame 238 -> 210 us in a stream; 24 sessions in 512^3
// f16+u16, 1200 -> 785 us of raycast kernel for a launch of 47 us.  The launch is bound by a surface's
// candidates lying in few threads' units, hence the packing; tiles of 8 and 32 pixels were within 2 %.
//
// A range image holds near depths as max over ~bits(z) and far depths as max over bits(z), so zero
// words mean "no brick"; its last two words are for bricks that reach behind the camera and have no
// image, and count for every tile.

struct RangeView {
    float P[9], o[3];    // P (p - o) = (u z, v z, z): level-0 image coordinates and camera depth
    int w, h, rgw, rgh;
    float min_d, max_d, vol_w;
    int n, nb;
    unsigned int* range;
};

__device__ __forceinline__ void range_add(unsigned int* at, float near_z, float far_z) {
    atomicMax(at, ~__float_as_uint(near_z));
    atomicMax(at + 1, __float_as_uint(far_z));
}

// One brick per lane, all lanes of the warp calling: `on` lanes hold a brick (bx, by, bz) of r whose
// bound can end large steps.  Its box -- the texel coordinates of the samples whose base voxel lies
// in it, from its first voxel to the next brick's, half a texel more at the volume's low edge, where
// coordinates clamp -- is widened by a margin above the rounding of a sample's position and
// projected.  Boxes of a few tiles are written by their lane; a box of many (coarse volumes: a brick
// of 25 cm covers some 30 tiles) by the whole warp.
__device__ __forceinline__ void range_bricks(const RangeView& r, bool on, int bx, int by, int bz) {
    int x0 = 0, x1 = -1, y0 = 0, y1 = -1;
    float zmin = 3.0e38f, zmax = -3.0e38f;
    if (on) {
        const float vox = r.vol_w / float(r.n), mid = 0.5f * float(r.n) - 0.5f;
        const float mar = 0.05f * vox + 4e-6f * (r.max_d + fabsf(r.o[0]) + fabsf(r.o[1]) + fabsf(r.o[2]));
        const float lx = (float(8 * bx) - (bx ? 0.f : 0.5f) - mid) * vox - mar - r.o[0];
        const float ly = (float(8 * by) - (by ? 0.f : 0.5f) - mid) * vox - mar - r.o[1];
        const float lz = (float(8 * bz) - (bz ? 0.f : 0.5f) - mid) * vox - mar - r.o[2];
        const float hx = (float(8 * bx + 8) - mid) * vox + mar - r.o[0];
        const float hy = (float(8 * by + 8) - mid) * vox + mar - r.o[1];
        const float hz = (float(8 * bz + 8) - mid) * vox + mar - r.o[2];
        float umin = 3.0e38f, umax = -3.0e38f, vmin = 3.0e38f, vmax = -3.0e38f;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const F3 q = mv3(r.P, F3{c & 1 ? hx : lx, c & 2 ? hy : ly, c & 4 ? hz : lz});
            const float iz = __fdividef(1.0f, q.z);
            zmin = fminf(zmin, q.z);
            zmax = fmaxf(zmax, q.z);
            umin = fminf(umin, q.x * iz);
            umax = fmaxf(umax, q.x * iz);
            vmin = fminf(vmin, q.y * iz);
            vmax = fmaxf(vmax, q.y * iz);
        }
        if (zmax >= r.min_d && zmin <= r.max_d) {
            // 0.1 px covers the rounding of the rays' and the corners' projections
            umin -= 0.1f; vmin -= 0.1f; umax += 0.1f; vmax += 0.1f;
            if (!(zmin > 1e-3f)) {   // reaches the camera plane: no image
                range_add(r.range + 2 * r.rgw * r.rgh, 0.0f, fmaxf(zmax, 0.0f));
            } else if (umax >= 0.f && vmax >= 0.f && umin <= float(r.w) && vmin <= float(r.h)) {
                x0 = int(fmaxf(umin, 0.f)) / kRangeTile;
                x1 = min(int(fminf(umax, float(r.w))) / kRangeTile, r.rgw - 1);
                y0 = int(fmaxf(vmin, 0.f)) / kRangeTile;
                y1 = min(int(fminf(vmax, float(r.h))) / kRangeTile, r.rgh - 1);
            }
        }
    }
    const int tiles = (x1 - x0 + 1) * (y1 - y0 + 1);
    unsigned int big = __ballot_sync(0xffffffffu, tiles > 16);
    if (tiles <= 16)
        for (int y = y0; y <= y1; ++y)
            for (int x = x0; x <= x1; ++x) range_add(r.range + 2 * (y * r.rgw + x), zmin, zmax);
    while (big) {
        const int from = __ffs(big) - 1;
        big &= big - 1;
        const int bx0 = __shfl_sync(0xffffffffu, x0, from), by0 = __shfl_sync(0xffffffffu, y0, from);
        const int bw = __shfl_sync(0xffffffffu, x1, from) - bx0 + 1, bt = __shfl_sync(0xffffffffu, tiles, from);
        const float bn = __shfl_sync(0xffffffffu, zmin, from), bf = __shfl_sync(0xffffffffu, zmax, from);
        const int rgw = __shfl_sync(0xffffffffu, r.rgw, from);
        unsigned int* const range = reinterpret_cast<unsigned int*>(
            __shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(r.range), from));
        for (int q = threadIdx.x & 31; q < bt; q += 32) range_add(range + 2 * ((by0 + q / bw) * rgw + bx0 + q % bw), bn, bf);
    }
}

// which of fusion unit u's four bricks (along x) have a bound that can end large steps
__device__ __forceinline__ unsigned int range_candidates(int n, int nb, const int* __restrict__ bdil, int u) {
    const int ux = (n + 31) >> 5, uy = n >> 3;
    const int bx = (u % ux) * 4, byz = u / ux, by = byz % uy, bz = byz / uy;
    const int* b = bdil + (bz * nb + by) * nb + bx;
    const int thr = __float_as_int(kSkipLarge);
    if ((nb & 3) == 0) {   // rows of bounds start on 16 bytes
        const int4 k = __ldg(reinterpret_cast<const int4*>(b));
        return (k.x < thr ? 1u : 0u) | (k.y < thr ? 2u : 0u) | (k.z < thr ? 4u : 0u) | (k.w < thr ? 8u : 0u);
    }
    unsigned int m = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q)
        if (bx + q < nb && __ldg(b + q) < thr) m |= 1u << q;
    return m;
}

// march state: everything the reference's loop carries from one sample to the next
struct RayState {
    float t;          // position of the next sample: base + idx * inc, one rounding
    float base;       // start of the current phase of the march
    float prev, prev_t, near_d, far_d;
    int idx;          // index of the next sample within the phase
    int small;        // 0 while stepping by 1.99 mu, 1 once stepping by 0.1 mu
    int prev_known;   // 0 when the last non-negative sample was skipped (value not computed)
    int guard;        // samples taken (hard bound)
    int sw;           // (samples taken when large steps ended) << 2 | how: 1 below 0.99, 2 negative
};

// position of sample k of the phase that starts at base
__device__ __forceinline__ float march_pos(float base, int k, float inc) { return __fmaf_rn(float(k), inc, base); }

// enter small steps: the next sample is base + inc (the sample that left large steps, or
// t - mu after a back-off, is the new base)
__device__ __forceinline__ void begin_small(RayState& st, float base, float small) {
    st.small = 1;
    st.base = base;
    st.idx = 1;
    st.t = march_pos(base, 1, small);
}

// The march's decision trace of one ray (written only in debug mode), so that a test can tell
// rays whose march took the same decisions as another implementation's from rays where a sample
// near 0.99 or 0 decided differently:
//   bits 40..  samples taken when the march left large steps (0: it never did)
//   bits  8..39 samples taken when the march ended (skipped samples count as taken, and so do those
//               left to the far plane where a depth range ended the ray: count_tails_kernel)
//   bits  4..5  how it left large steps: 1 a sample in [0, 0.99), 2 a negative one (back-off)
//   bits  0..1  how it ended: 0 past the far plane or the sample bound, 1 negative first
//               sample, 2 refined hit
// A ray that returns before marching has trace 0.
__device__ __forceinline__ unsigned long long ray_trace_code(const RayState& st, float precise) {
    const int end = precise != 0.0f ? 2 : (st.t < st.far_d && st.guard < kMaxMarchSamples ? 1 : 0);
    return (static_cast<unsigned long long>(st.sw >> 2) << 40) | (static_cast<unsigned long long>(st.guard) << 8) |
           static_cast<unsigned long long>((st.sw & 3) << 4) | static_cast<unsigned long long>(end);
}

// Work counts of the march, kept only by the kernels' counting instantiation (debug mode
// KF_DEBUG_COUNTERS); the production instantiation compiles every count away.
enum RayCount {
    kCntRays = 0,        // rays that marched
    kCntEvalLarge,       // samples evaluated (trilinear) during large steps
    kCntEvalSmall,       // samples evaluated during small steps
    kCntSkips,           // cell skips (each jumps over one or more samples)
    kCntSkipped,         // samples jumped over by the skips
    kCntGrad,            // gradient samples of hits (six per refined hit)
    kCntQueued,          // rays handed from a lane to the long-ray warp kernel
    kCntRounds,          // warp rounds of the long-ray kernel (32 or 64 samples each)
    kRayCounts
};

template <bool kOn> struct MarchCount {
    static constexpr bool on = false;
    __device__ __forceinline__ void add(int, unsigned int) {}
    __device__ __forceinline__ void flush(unsigned long long*) {}
};
template <> struct MarchCount<true> {
    static constexpr bool on = true;
    unsigned int c[kRayCounts] = {};
    __device__ __forceinline__ void add(int k, unsigned int x) { c[k] += x; }
    __device__ __forceinline__ void flush(unsigned long long* dst) {
        if (!dst) return;
#pragma unroll
        for (int k = 0; k < kRayCounts; ++k)
            if (c[k]) atomicAdd(dst + k, static_cast<unsigned long long>(c[k]));
    }
};

// a ray handed from a lane to a warp: where it is, its exact march state and its geometry (so
// the warp neither reloads the pose nor divides again)
struct __align__(16) LongRay {
    int s, level, i, j;
    RayState st;
    RayGeo g;
};

__device__ __forceinline__ void ray_matrix(const SessionDev* S, const LevelDev& Lv, float* m, F3& o) {
    // R_prev * K_l^-1 (the reference forms mat3(pose) * invK per ray), each product and sum
    // rounded on its own -- the same arithmetic as the host's for the stage raycast, so that a
    // stage raycast of a session's volume at its pose takes the session's rays bit for bit
    const float* R = S->pose->Rpf;
#pragma unroll
    for (int col = 0; col < 3; ++col)
#pragma unroll
        for (int row = 0; row < 3; ++row)
            m[col * 3 + row] = __fadd_rn(__fadd_rn(__fmul_rn(R[row], Lv.ik[col * 3 + 0]),
                                                   __fmul_rn(R[3 + row], Lv.ik[col * 3 + 1])),
                                         __fmul_rn(R[6 + row], Lv.ik[col * 3 + 2]));
    o = F3{S->pose->tpf[0], S->pose->tpf[1], S->pose->tpf[2]};
}

// ray through pixel (i, j): direction (R K^-1)(i + .5, j + .5, 1), not normalised, so t is
// camera depth
__device__ __forceinline__ void make_geo(const SessionDev* S, const float* m, F3 o, int i, int j, RayGeo& g) {
    g.o = o;
    g.dir = mv3(m, F3{float(i) + 0.5f, float(j) + 0.5f, 1.0f});
    g.sc = float(S->n) / S->vol_w;
    g.off = 0.5f * float(S->n) - 0.5f;
    g.tox = o.x * g.sc + g.off; g.toy = o.y * g.sc + g.off; g.toz = o.z * g.sc + g.off;
    g.tdx = g.dir.x * g.sc; g.tdy = g.dir.y * g.sc; g.tdz = g.dir.z * g.sc;
    // only the skips' cell exits use these, 0.01 texel inside the faces: the fast reciprocal's
    // 2 ulp cannot move a skip across a sample
    g.itdx = __fdividef(1.0f, g.tdx); g.itdy = __fdividef(1.0f, g.tdy); g.itdz = __fdividef(1.0f, g.tdz);
}

// texel coordinate of the sample at t, (o + dir t) * sc + off, with its roundings spelled out
// (two fused multiply-adds): a sample's value must not depend on which kernel, or which
// branch of the march, evaluates it, since its comparison with 0.99 or 0 decides the march
__device__ __forceinline__ void texel(const RayGeo& g, float t, float& x, float& y, float& z) {
    x = __fmaf_rn(__fmaf_rn(g.dir.x, t, g.o.x), g.sc, g.off);
    y = __fmaf_rn(__fmaf_rn(g.dir.y, t, g.o.y), g.sc, g.off);
    z = __fmaf_rn(__fmaf_rn(g.dir.z, t, g.o.z), g.sc, g.off);
}

__device__ __forceinline__ void clamp_voxel(int n, int& x, int& y, int& z) {
    x = min(max(x, 0), n - 1);
    y = min(max(y, 0), n - 1);
    z = min(max(z, 0), n - 1);
}

__device__ __forceinline__ unsigned int voxel_index(unsigned int n, int x, int y, int z) {
    return (unsigned(z) * n + unsigned(y)) * n + unsigned(x);
}

template <class TF>
__device__ __forceinline__ float sample_at(const SessionDev* S, const RayGeo& g, const TF* f, float t) {
    float x, y, z;
    texel(g, t, x, y, z);
    const InnerBase b = inner_base(S->n, x, y, z);
    if (b.in) return trilinear_inner(f, unsigned(S->n), voxel_index(unsigned(S->n), b.x0, b.y0, b.z0), b.ax, b.ay, b.az);
    return trilinear(f, S->n, x, y, z);
}

// intersectBBox and the [min, max] depth clip; false when the reference returns before
// marching (such rays keep the previous map contents unless keep_on_miss is off)
__device__ __forceinline__ bool ray_start(const SessionDev* S, const RayGeo& g, RayState& st) {
    const F3 inv{1.0f / g.dir.x, 1.0f / g.dir.y, 1.0f / g.dir.z};
    const float half = S->vol_w * 0.5f;
    const F3 o = g.o;
    const float t0x = (-half - o.x) * inv.x, t1x = (half - o.x) * inv.x;
    const float t0y = (-half - o.y) * inv.y, t1y = (half - o.y) * inv.y;
    const float t0z = (-half - o.z) * inv.z, t1z = (half - o.z) * inv.z;
    float tmin = fminf(t0x, t1x), tmax = fmaxf(t0x, t1x);
    tmin = fmaxf(tmin, fminf(t0y, t1y));
    tmax = fminf(tmax, fmaxf(t0y, t1y));
    tmin = fmaxf(tmin, fminf(t0z, t1z));
    tmax = fminf(tmax, fmaxf(t0z, t1z));
    if (tmax < tmin) { tmin = -1.0f; tmax = -1.0f; }
    if (tmax < 0.0f) return false;
    const float near_d = fmaxf(S->min_d, tmin), far_d = fminf(S->max_d, tmax);
    if (near_d >= far_d) return false;
    st.t = near_d;
    st.base = near_d;
    st.idx = 0;
    st.near_d = near_d;
    st.far_d = far_d;
    st.prev = 0.f;
    st.prev_t = 0.f;
    st.small = 0;
    st.prev_known = 1;
    st.guard = 0;
    st.sw = 0;
    return true;
}

// t at which the base voxel of the march leaves the voxel box [lo, hi) per axis (0.01 texel
// inside its faces); faces on the volume's edge do not bound (coordinates clamp there).  The
// margin absorbs the rounding of the affine form to + td t: a skip that stops early only
// evaluates samples it could have skipped; it never passes a sample outside the box.
__device__ __forceinline__ float box_exit(const RayGeo& g, int n, int lox, int hix, int loy, int hiy, int loz, int hiz,
                                          float t_far) {
    float t = t_far;
    if (g.tdx > 0.f && hix < n) t = fminf(t, (float(hix) - 0.01f - g.tox) * g.itdx);
    if (g.tdx < 0.f && lox > 0) t = fminf(t, (float(lox) + 0.01f - g.tox) * g.itdx);
    if (g.tdy > 0.f && hiy < n) t = fminf(t, (float(hiy) - 0.01f - g.toy) * g.itdy);
    if (g.tdy < 0.f && loy > 0) t = fminf(t, (float(loy) + 0.01f - g.toy) * g.itdy);
    if (g.tdz > 0.f && hiz < n) t = fminf(t, (float(hiz) - 0.01f - g.toz) * g.itdz);
    if (g.tdz < 0.f && loz > 0) t = fminf(t, (float(loz) + 0.01f - g.toz) * g.itdz);
    return t;
}

// The run of consecutive skippable super-bricks the ray is in, from super-brick s (skippable):
// the t before which every sample's base voxel lies in the run.  Per axis, tc is the t at
// which the ray crosses the cell's face ahead and tm the t at which it comes within 0.01 texel
// of it (faces on the volume's edge do not bound: coordinates clamp there).  The ray leaves a
// cell through the face it crosses first; the run continues into the neighbour across that
// face when the neighbour is skippable and the crossing is clean -- every other coordinate
// still 0.01 texel inside the cell's faces ahead at that t, so a rounded sample near the
// crossing lies in one of the two cells and in no third one.  The run ends at the last cell's
// margined exit, exactly where a skip of that cell alone would end.  At most kRunCells cells.
__device__ __forceinline__ void cell_face(float to, float td, float itd, int s, int n, float t_far, float& tc,
                                          float& tm) {
    // the face of super-brick s ahead along one axis: crossing t and margined t
    tc = tm = t_far;
    if (td > 0.f && 32 * (s + 1) < n) {
        const float face = float(32 * (s + 1));
        tc = (face - to) * itd;
        tm = (face - 0.01f - to) * itd;
    } else if (td < 0.f && s > 0) {
        const float face = float(32 * s);
        tc = (face - to) * itd;
        tm = (face + 0.01f - to) * itd;
    }
}

__device__ __forceinline__ float superbrick_run_exit(const SessionDev* S, const RayGeo& g, int thr, int sx, int sy,
                                                     int sz, float t_far) {
    const int n = S->n, ns = S->ns;
    float tcx, tmx, tcy, tmy, tcz, tmz;
    cell_face(g.tox, g.tdx, g.itdx, sx, n, t_far, tcx, tmx);
    cell_face(g.toy, g.tdy, g.itdy, sy, n, t_far, tcy, tmy);
    cell_face(g.toz, g.tdz, g.itdz, sz, n, t_far, tcz, tmz);
    for (int step = 0; step < kRunCells - 1; ++step) {
        if (tcx <= tcy && tcx <= tcz) {          // leaves through the x face
            if (!(tcx < t_far) || tmy < tcx || tmz < tcx) break;
            const int nx = sx + (g.tdx > 0.f ? 1 : -1);
            if (__ldg(S->sdil + (sz * ns + sy) * ns + nx) < thr) break;
            sx = nx;
            cell_face(g.tox, g.tdx, g.itdx, sx, n, t_far, tcx, tmx);
        } else if (tcy <= tcz) {                 // the y face
            if (!(tcy < t_far) || tmx < tcy || tmz < tcy) break;
            const int ny = sy + (g.tdy > 0.f ? 1 : -1);
            if (__ldg(S->sdil + (sz * ns + ny) * ns + sx) < thr) break;
            sy = ny;
            cell_face(g.toy, g.tdy, g.itdy, sy, n, t_far, tcy, tmy);
        } else {                                 // the z face
            if (!(tcz < t_far) || tmx < tcz || tmy < tcz) break;
            const int nz = sz + (g.tdz > 0.f ? 1 : -1);
            if (__ldg(S->sdil + (nz * ns + sy) * ns + sx) < thr) break;
            sz = nz;
            cell_face(g.toz, g.tdz, g.itdz, sz, n, t_far, tcz, tmz);
        }
    }
    return fminf(fminf(tmx, tmy), tmz);
}

// a read-only load the compiler keeps where it is written (not sunk into a branch)
__device__ __forceinline__ int ld_keep(const int* p) {
    int v;
    asm volatile("ld.global.nc.s32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

// Skip the sample at st.t and every later one before lim: the next sample is the first index
// k > idx with base + k inc >= lim (positions increase with k), or the last index the sample bound
// allows.
__device__ __forceinline__ void skip_to(RayState& st, float lim, float inc) {
    const int k_lo = st.idx + 1, k_hi = st.idx + (kMaxMarchSamples - st.guard);
    int k = k_lo;
    const float est = __fdividef(lim - st.base, inc);   // within an index or two of the answer
    if (est > float(k_lo)) k = int(fminf(est, float(k_hi)));
    while (k > k_lo && !(march_pos(st.base, k - 1, inc) < lim)) --k;
    while (k < k_hi && march_pos(st.base, k, inc) < lim) ++k;
    st.guard += k - st.idx;
    st.idx = k;
    st.prev_t = march_pos(st.base, k - 1, inc);
    st.t = march_pos(st.base, k, inc);
    st.prev_known = 0;
}

// Samples whose base voxel lies in a cell whose distance lower bound is at or above the
// current threshold (0.991 during large steps, 0.001 during small steps) cannot change the
// march.  If the sample at st.t, with base voxel (vx, vy, vz), is such a sample, advance st past
// every following sample in the same cell -- the run of skippable 32^3 super-bricks along the
// ray when its super-brick qualifies, else its 8^3 brick -- to the first sample index whose
// position is at or past the cell's (run's) exit, and return true.  The brick's bound decides (a
// super-brick's is the minimum over its bricks', so a skippable super-brick has no other).  The
// super-brick's is read by a skip only, since with the depth ranges most iterations evaluate their
// sample; kEager reads it beside the brick's, in one round trip, where latency bounds the march (a
// single session: 38 us against 42 for 320x240 in 128^3).  With the taps' and the gradient's shared
// arithmetic and a kernel per volume format the raycast of 24 full-size sessions went from 785 to
// 671 us.
template <bool kEager>
__device__ __forceinline__ bool skip_cell(const SessionDev* S, const RayGeo& g, RayState& st, int vx, int vy, int vz,
                                          float inc) {
    // order-preserving int keys of the two thresholds
    const int thr = st.small ? __float_as_int(kSkipSmall) : __float_as_int(kSkipLarge);
    const int nb = S->nb, bx = vx >> 3, by = vy >> 3, bz = vz >> 3;   // (n / 8)^3 bricks: 32-bit indices
    int early = 0;
    if constexpr (kEager) early = ld_keep(S->sdil + ((vz >> 5) * S->ns + (vy >> 5)) * S->ns + (vx >> 5));
    if (__ldg(S->bdil + (bz * nb + by) * nb + bx) < thr) return false;
    const int n = S->n, ns = S->ns, sx = vx >> 5, sy = vy >> 5, sz = vz >> 5;
    const float exit_t = (kEager ? early : __ldg(S->sdil + (sz * ns + sy) * ns + sx)) >= thr
                             ? superbrick_run_exit(S, g, thr, sx, sy, sz, st.far_d)
                             : box_exit(g, n, bx * 8, bx * 8 + 8, by * 8, by * 8 + 8, bz * 8, bz * 8 + 8, st.far_d);
    // skip this sample and every later one whose base voxel stays in the box
    skip_to(st, fminf(exit_t, st.far_d), inc);
    return true;
}

// The reference's march loop for one lane (project/src/raycast.cu:75-117).  Returns 1 when
// the ray is finished (precise = refined hit distance, 0 for none) and 0 when `budget`
// iterations ran out with the ray still marching (state kept in st).
template <class TF, class Cnt, bool kEager>
__device__ int march_serial(const SessionDev* S, const RayGeo& g, const TF* f, RayState& st, int budget,
                            float& precise, Cnt& cnt) {
    const int n = S->n;
    const float mu = S->mu, large = mu * S->step_l, small = mu * S->step_s;
    const int* __restrict__ bdil = S->bdil;
    int iters = 0;
    while (st.t < st.far_d && st.guard < kMaxMarchSamples) {
        if (iters++ >= budget) return 0;
        const float inc = st.small ? small : large;
        float x, y, z;
        texel(g, st.t, x, y, z);
        const InnerBase b = inner_base(n, x, y, z);
        const int g0 = st.guard;
        bool skipped;
        if constexpr (kEager) {
            int vx = b.x0, vy = b.y0, vz = b.z0;
            if (!b.in) clamp_voxel(n, vx, vy, vz);
            skipped = bdil && skip_cell<true>(S, g, st, vx, vy, vz, inc);
        } else {   // in 64 registers two copies of the skip spill less than clamped copies of the voxel
            skipped = false;
            if (bdil) {
                if (b.in) {
                    skipped = skip_cell<false>(S, g, st, b.x0, b.y0, b.z0, inc);
                } else {
                    const TexelBase tb = texel_base(n, x, y, z);
                    skipped = skip_cell<false>(S, g, st, tb.x0, tb.y0, tb.z0, inc);
                }
            }
        }
        if (skipped) {
            cnt.add(kCntSkips, 1u);
            cnt.add(kCntSkipped, unsigned(st.guard - g0));
            continue;
        }
        const float tsdf = b.in ? trilinear_inner(f, unsigned(n), voxel_index(unsigned(n), b.x0, b.y0, b.z0), b.ax, b.ay, b.az)
                                : trilinear(f, n, x, y, z);
        cnt.add(st.small ? kCntEvalSmall : kCntEvalLarge, 1u);
        ++st.guard;
        if (tsdf < 0.0f) {
            if (st.t != st.near_d) {
                if (!st.small) {   // went through the surface with a large step: back off by mu
                    st.sw = (st.guard << 2) | 2;
                    begin_small(st, __fsub_rn(st.t, mu), small);
                    continue;
                }
                if (!st.prev_known) st.prev = sample_at(S, g, f, st.prev_t);
                precise = st.t - small * st.prev / (tsdf - st.prev);   // the reference's formula
            }
            return 1;
        }
        st.prev = tsdf;
        st.prev_known = 1;
        st.prev_t = st.t;
        if (!st.small && tsdf < 0.99f) {   // the region of uncertainty: small steps from here
            st.sw = (st.guard << 2) | 1;
            begin_small(st, st.t, small);
        } else {
            ++st.idx;
            st.t = march_pos(st.base, st.idx, inc);
        }
    }
    return 1;
}

// The same loop for one ray, carried by all 32 lanes of a warp (every lane holds the same
// g and st): each round lane k evaluates the sample k indices ahead, and the first sample
// that changes the state -- a negative value, or below 0.99 during large steps -- is applied.
// A round that follows a round without any such sample takes two sets, samples k and 32 + k
// (such rays are in a long run of samples that change nothing, a grazing ray in small steps
// for instance); the first event in sample order is applied all the same.
template <class TF, class Cnt>
__device__ void march_coop(const SessionDev* S, const RayGeo& g, const TF* f, RayState& st, int lane,
                           float& precise, Cnt& cnt) {
    const float mu = S->mu, large = mu * S->step_l, small = mu * S->step_s;
    const unsigned int full = 0xffffffffu;
    bool wide = false;   // the last round changed nothing
    while (st.t < st.far_d && st.guard < kMaxMarchSamples) {
        const float inc = st.small ? small : large;
        if (S->bdil) {
            float x, y, z;
            texel(g, st.t, x, y, z);
            const InnerBase b = inner_base(S->n, x, y, z);
            int vx = b.x0, vy = b.y0, vz = b.z0;
            if (!b.in) clamp_voxel(S->n, vx, vy, vz);
            const int g0 = st.guard;
            if (skip_cell<true>(S, g, st, vx, vy, vz, inc)) {   // every lane takes the same steps
                if (lane == 0) {
                    cnt.add(kCntSkips, 1u);
                    cnt.add(kCntSkipped, unsigned(st.guard - g0));
                }
                wide = false;
                continue;
            }
        }
        float tk[2], fk[2];
        bool valid[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int n = 32 * j + lane;   // sample n of the round
            tk[j] = march_pos(st.base, st.idx + n, inc);
            valid[j] = (j == 0 || wide) && tk[j] < st.far_d && st.guard + n < kMaxMarchSamples;
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            fk[j] = valid[j] ? sample_at(S, g, f, tk[j]) : 0.0f;
            if (valid[j]) cnt.add(st.small ? kCntEvalSmall : kCntEvalLarge, 1u);
        }
        if (lane == 0) cnt.add(kCntRounds, 1u);
        unsigned int evm[2], valm[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            evm[j] = __ballot_sync(full, valid[j] && (fk[j] < 0.0f || (!st.small && fk[j] < 0.99f)));
            valm[j] = __ballot_sync(full, valid[j]);   // valid samples form a prefix in n
        }
        if (!evm[0] && !evm[1]) {
            if (!valm[0]) break;
            const int js = valm[1] ? 1 : 0;
            const int last = 31 - __clz(js ? valm[1] : valm[0]);
            st.prev = __shfl_sync(full, js ? fk[1] : fk[0], last);
            st.prev_t = __shfl_sync(full, js ? tk[1] : tk[0], last);
            st.prev_known = 1;
            st.guard += 32 * js + last + 1;
            st.idx += 32 * js + last + 1;
            st.t = march_pos(st.base, st.idx, inc);
            wide = true;
            continue;
        }
        wide = false;
        const int js = evm[0] ? 0 : 1;
        const float tj = js ? tk[1] : tk[0], fj = js ? fk[1] : fk[0];
        const int e = __ffs(js ? evm[1] : evm[0]) - 1;
        const float te = __shfl_sync(full, tj, e), fe = __shfl_sync(full, fj, e);
        // the sample before the event: lane e - 1 of the same set, or the first set's last lane
        const float tb = __shfl_sync(full, tj, max(e - 1, 0)), fb = __shfl_sync(full, fj, max(e - 1, 0));
        const float tb0 = __shfl_sync(full, tk[0], 31), fb0 = __shfl_sync(full, fk[0], 31);
        const int ne = 32 * js + e;
        if (ne > 0) {
            st.prev = e > 0 ? fb : fb0;
            st.prev_t = e > 0 ? tb : tb0;
            st.prev_known = 1;
        }
        st.guard += ne + 1;
        if (fe < 0.0f) {
            if (te != st.near_d) {
                if (!st.small) {
                    st.sw = (st.guard << 2) | 2;
                    begin_small(st, __fsub_rn(te, mu), small);
                    continue;
                }
                if (!st.prev_known) st.prev = sample_at(S, g, f, st.prev_t);
                precise = te - small * st.prev / (fe - st.prev);
            }
            return;
        }
        st.sw = (st.guard << 2) | 1;   // 0 <= fe < 0.99 during large steps (only they are events)
        st.prev = fe;
        st.prev_t = te;
        st.prev_known = 1;
        begin_small(st, te, small);
    }
}

// Start and end the ray of pixel (i, j) of a level by its tile's depth range: past every sample
// that no brick with a low bound can hold.
template <class Cnt>
__device__ __forceinline__ void clip_to_range(const SessionDev* S, int level, int i, int j, RayState& st, Cnt& cnt) {
    const int x = ((i + 1) << level) - 1, y = ((j + 1) << level) - 1;   // the level-0 pixel it passes through
    const uint2* r = reinterpret_cast<const uint2*>(S->range);
    const uint2 tile = __ldg(r + (y / kRangeTile) * S->rgw + x / kRangeTile), all = __ldg(r + S->rgw * S->rgh);
    const unsigned int near_k = max(tile.x, all.x), far_k = max(tile.y, all.y);
    // no brick: nothing to meet before the far plane
    const float lim = near_k ? __uint_as_float(~near_k) : st.far_d;
    if (st.t < lim) {
        const int g0 = st.guard;
        skip_to(st, fminf(lim, st.far_d), S->mu * S->step_l);
        cnt.add(kCntSkips, 1u);
        cnt.add(kCntSkipped, unsigned(st.guard - g0));
    }
    st.far_d = fminf(st.far_d, near_k ? __uint_as_float(far_k) : st.t);
}

// computeGradient (project/src/raycast.cu:29-42) at the hit: texel coordinates of the hit
// and the offset of the six central-difference samples (mu / 2 apart, in uvw units)
struct HitGeo {
    F3 vtx;
    float x, y, z, rt, r;
};

__device__ __forceinline__ HitGeo hit_geo(const SessionDev* S, const RayGeo& g, float precise) {
    HitGeo h;
    h.vtx = F3{__fmaf_rn(g.dir.x, precise, g.o.x), __fmaf_rn(g.dir.y, precise, g.o.y),
               __fmaf_rn(g.dir.z, precise, g.o.z)};
    h.r = S->mu * 0.5f / S->vol_w;
    h.rt = h.r * float(S->n);
    h.x = __fmaf_rn(h.vtx.x, g.sc, g.off);
    h.y = __fmaf_rn(h.vtx.y, g.sc, g.off);
    h.z = __fmaf_rn(h.vtx.z, g.sc, g.off);
    return h;
}

// gradient sample q of computeGradient: q = 0, 1, 2 at +rt along x, y, z; 3, 4, 5 at -rt
template <class TF>
__device__ __forceinline__ float grad_sample(const TF* f, int n, const HitGeo& h, int q) {
    const float d = q < 3 ? h.rt : -h.rt;
    const int a = q < 3 ? q : q - 3;
    return trilinear(f, n, a == 0 ? __fadd_rn(h.x, d) : h.x, a == 1 ? __fadd_rn(h.y, d) : h.y,
                     a == 2 ? __fadd_rn(h.z, d) : h.z);
}

// The six samples of a hit whose taps all lie inside the volume (almost every one) share the base
// voxel and the weights of the two axes they do not move along, and clamp nothing; the others take
// grad_sample's general form.
template <class TF>
__device__ __forceinline__ void grad_samples(const TF* f, int n, const HitGeo& h, float (&v)[6]) {
    const InnerBase b = inner_base(n, h.x, h.y, h.z);
    float ax[6];
    int d[6];   // base voxel of sample q along its axis
    unsigned int far = 0;
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        const int a = q < 3 ? q : q - 3;
        d[q] = floor_split(__fadd_rn(a == 0 ? h.x : a == 1 ? h.y : h.z, q < 3 ? h.rt : -h.rt), ax[q]);
        far = max(far, unsigned(d[q]));
    }
    if (b.in && far < unsigned(n - 1)) {
        const unsigned int un = unsigned(n), idx = voxel_index(un, b.x0, b.y0, b.z0);
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            const int a = q < 3 ? q : q - 3;
            const unsigned int at = idx + unsigned(d[q] - (a == 0 ? b.x0 : a == 1 ? b.y0 : b.z0)) * (a == 0 ? 1u : a == 1 ? un : un * un);
            v[q] = trilinear_inner(f, un, at, a == 0 ? ax[q] : b.ax, a == 1 ? ax[q] : b.ay, a == 2 ? ax[q] : b.az);
        }
        return;
    }
#pragma unroll 1
    for (int q = 0; q < 6; ++q) {
        const float w = grad_sample(f, n, h, q);
#pragma unroll
        for (int k = 0; k < 6; ++k)
            if (k == q) v[k] = w;
    }
}

// the normal from the six samples and the map writes (project/src/raycast.cu:120-144)
__device__ __forceinline__ void write_hit(const SessionDev* S, int level, int i, int j, bool hit, const HitGeo& h,
                                          const float (&v)[6]) {
    const int w = S->lv[level].w;
    float4* ov = S->pv[level] + size_t(j) * w + i;
    float4* on = S->pn[level] + size_t(j) * w + i;
    if (hit) {
        F3 gr{(v[3] - v[0]) / h.r, (v[4] - v[1]) / h.r, (v[5] - v[2]) / h.r};
        const float gn = sqrtf(dot3(gr, gr));
        if (depth_valid(gn)) {
            gr = F3{gr.x / gn, gr.y / gn, gr.z / gn};
            *ov = make_float4(h.vtx.x, h.vtx.y, h.vtx.z, kValid);
            *on = make_float4(gr.x, gr.y, gr.z, kValid);
            return;
        }
    }
    *ov = make_float4(0.f, 0.f, 0.f, kInvalid);
    *on = make_float4(0.f, 0.f, 0.f, kInvalid);
}

__device__ __forceinline__ void write_trace(const SessionDev* S, int level, int i, int j, unsigned long long code) {
    unsigned long long* tr = S->trace[level];
    if (tr) tr[size_t(j) * S->lv[level].w + i] = code;
}

// the work counts' share of the samples between the end of a ray's depth range and its far plane
template <class Cnt>
__device__ __forceinline__ void count_tail(const SessionDev* S, const RayGeo& g, float precise, RayState st, Cnt& cnt) {
    if constexpr (Cnt::on) {
        RayState whole;
        if (!S->range || precise != 0.0f || st.t < st.far_d || !ray_start(S, g, whole)) return;
        if (!(st.t < whole.far_d) || st.guard >= kMaxMarchSamples) return;
        const int g0 = st.guard;
        skip_to(st, whole.far_d, S->mu * (st.small ? S->step_s : S->step_l));
        cnt.add(kCntSkipped, unsigned(st.guard - g0));
    }
}

template <class TF, class Cnt>
__device__ void finish_ray(const SessionDev* S, const RayGeo& g, const TF* f, int level, int i, int j, float precise,
                           const RayState& st, Cnt& cnt) {
    write_trace(S, level, i, j, ray_trace_code(st, precise));
    count_tail(S, g, precise, st, cnt);
    const HitGeo h = hit_geo(S, g, precise);
    float v[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (precise != 0.0f) {
        cnt.add(kCntGrad, 6u);
        grad_samples(f, S->n, h, v);
    }
    write_hit(S, level, i, j, precise != 0.0f, h, v);
}

// the same for a ray carried by a whole warp: lanes 0-5 take one gradient sample each, lane 0
// writes
template <class TF, class Cnt>
__device__ void finish_ray_warp(const SessionDev* S, const RayGeo& g, const TF* f, int level, int i, int j,
                                float precise, int lane, const RayState& st, Cnt& cnt) {
    if (lane == 0) {
        write_trace(S, level, i, j, ray_trace_code(st, precise));
        count_tail(S, g, precise, st, cnt);
    }
    const HitGeo h = hit_geo(S, g, precise);
    float mine = 0.f;
    if (precise != 0.0f && lane < 6) {
        mine = grad_sample(f, S->n, h, lane);
        cnt.add(kCntGrad, 1u);
    }
    float v[6];
#pragma unroll
    for (int q = 0; q < 6; ++q) v[q] = __shfl_sync(0xffffffffu, mine, q);
    if (lane == 0) write_hit(S, level, i, j, precise != 0.0f, h, v);
}

__device__ __forceinline__ void write_miss(const SessionDev* S, int level, int i, int j) {
    write_trace(S, level, i, j, 0ull);
    if (S->keep_on_miss) return;
    const int w = S->lv[level].w;
    S->pv[level][size_t(j) * w + i] = make_float4(0.f, 0.f, 0.f, kInvalid);
    S->pn[level][size_t(j) * w + i] = make_float4(0.f, 0.f, 0.f, kInvalid);
}

// where lanes hand over the rays they do not finish
struct RayQueue {
    LongRay* rays;
    unsigned int* count;
    int cap;
};

template <class TF, class Cnt, bool kEager>
__device__ void serial_ray(const RayQueue& rq, const SessionDev* S, int s, const float* m, F3 o, int level, int i,
                           int j, int budget, Cnt& cnt) {
    const TF* f = static_cast<const TF*>(S->tf);
    RayGeo g;
    make_geo(S, m, o, i, j, g);
    RayState st;
    if (!ray_start(S, g, st)) {
        write_miss(S, level, i, j);
        return;
    }
    cnt.add(kCntRays, 1u);
    if (S->range) clip_to_range(S, level, i, j, st, cnt);
    float precise = 0.0f;
    if (!march_serial<TF, Cnt, kEager>(S, g, f, st, budget, precise, cnt)) {
        const unsigned int slot = atomicAdd(rq.count, 1u);
        if (slot < unsigned(rq.cap)) {
            rq.rays[slot] = LongRay{s, level, i, j, st, g};
            cnt.add(kCntQueued, 1u);
            return;
        }
        march_serial<TF, Cnt, kEager>(S, g, f, st, 0x7fffffff, precise, cnt);   // queue full: finish here
    }
    finish_ray(S, g, f, level, i, j, precise, st, cnt);
}

// The first launch of a step: clears the wait record and the counters, and makes the depth ranges of
// every session that raycasts in this step: a thread tests a fusion unit's four bricks, and the block's
// candidates are packed and projected one per thread.
__global__ void __launch_bounds__(256) ray_range_kernel(EngineView v) {
    if (blockIdx.x == 0) {
        if (threadIdx.x < sizeof(GridSync) / 4) reinterpret_cast<unsigned int*>(v.sync)[threadIdx.x] = 0u;
        if (threadIdx.x < kCounters) v.counters[threadIdx.x] = 0u;
    }
    __shared__ unsigned short list[256 * 4];
    __shared__ int packed;
    const int tid = threadIdx.x;
    const long long total = v.tb->fuse_total, stride = (long long)gridDim.x * blockDim.x;
    const int S_cap = v.tb->S;
    RangeView r;
    r.rgw = 0;
    r.range = nullptr;
    int cur = -1;
    bool has_inv = false;
    for (long long base = (long long)blockIdx.x * blockDim.x; base < total; base += stride) {
        unsigned int m = 0;
        if (base + tid < total) {
            const int s = unit_session(v.fuse_prefix, base + tid, S_cap);
            const SessionDev* S = &v.sess[s];
            const StepDev st = v.step[s];
            if (st.active && !st.first && S->range)
                m = range_candidates(S->n, S->nb, S->bdil, int(base + tid - __ldg(v.fuse_prefix + s)));
        }
        const int count = block_pack(m, list, &packed);
        for (int i = tid & ~31; i < count; i += 256) {
            bool on = i + (tid & 31) < count;
            int bx = 0, by = 0, bz = 0;
            if (on) {
                const int code = list[i + (tid & 31)];
                const long long g = base + (code >> 2);
                const int s = unit_session(v.fuse_prefix, g, S_cap);
                if (s != cur) {
                    const SessionDev* S = &v.sess[s];
                    const LevelDev& L = S->lv[0];
                    // the inverse of the pose's 3x3, adjugate over determinant (kf_set_pose takes
                    // matrices that are not exactly rotations, and the rays use them as they are)
                    float R[9], I[9];
#pragma unroll
                    for (int q = 0; q < 9; ++q) R[q] = S->pose->Rpf[q];   // camera -> world, column-major
                    I[0] = R[4] * R[8] - R[5] * R[7]; I[3] = R[5] * R[6] - R[3] * R[8]; I[6] = R[3] * R[7] - R[4] * R[6];
                    I[1] = R[2] * R[7] - R[1] * R[8]; I[4] = R[0] * R[8] - R[2] * R[6]; I[7] = R[1] * R[6] - R[0] * R[7];
                    I[2] = R[1] * R[5] - R[2] * R[4]; I[5] = R[2] * R[3] - R[0] * R[5]; I[8] = R[0] * R[4] - R[1] * R[3];
                    const float det = R[0] * I[0] + R[3] * I[1] + R[6] * I[2];
                    has_inv = fabsf(det) > 1e-3f;
                    const float od = 1.0f / det;
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        // column c of K R^-1
                        r.P[c * 3 + 0] = (L.fx * I[c * 3] + L.cx * I[c * 3 + 2]) * od;
                        r.P[c * 3 + 1] = (L.fy * I[c * 3 + 1] + L.cy * I[c * 3 + 2]) * od;
                        r.P[c * 3 + 2] = I[c * 3 + 2] * od;
                        r.o[c] = S->pose->tpf[c];
                    }
                    r.w = S->W; r.h = S->H; r.rgw = S->rgw; r.rgh = S->rgh;
                    r.min_d = S->min_d; r.max_d = S->max_d; r.vol_w = S->vol_w;
                    r.n = S->n; r.nb = S->nb;
                    r.range = S->range;
                    cur = s;
                }
                const int u = int(g - __ldg(v.fuse_prefix + s)), ux = (r.n + 31) >> 5;
                bx = (u % ux) * 4 + (code & 3);
                by = (u / ux) % r.nb;
                bz = u / (ux * r.nb);
                if (!has_inv) {   // no projection: every ray its whole length
                    range_add(r.range + 2 * r.rgw * r.rgh, 0.0f, 3.0e38f);
                    on = false;
                }
            }
            range_bricks(r, on, bx, by, bz);
        }
        __syncthreads();   // the list and its count are read before the next units' are written
    }
}

// Each warp pulls 8 x 4-ray tiles on its own (no block-wide barrier).  Steps of many ray tiles
// run four blocks per SM (64 registers: more warps to hide the gathers behind); a single
// session's step runs three (80 registers: fewer instructions per sample, a shorter tail).
template <int kBlocksPerSm, bool kCount, int kFmt>
__global__ void __launch_bounds__(256, kBlocksPerSm) raycast_kernel(EngineView v) {
    MarchCount<kCount> cnt;
    const int lane = threadIdx.x & 31;
    const int ntiles = v.tb->n_ray;
    const int budget = v.tb->ray_budget;
    const int tw = v.tb->ray_tw;
    const int lx = lane % tw, ly = lane / tw;
    const RayQueue rq{v.longq, v.counters + 6, v.longq_cap};
    while (true) {
        int t = 0;
        if (lane == 0) t = int(atomicAdd(&v.counters[0], 1u));
        t = __shfl_sync(0xffffffffu, t, 0);
        if (t >= ntiles) break;
        const RayTile T = v.ray[t];
        const StepDev st = v.step[T.s];
        if (!st.active || st.first) continue;
        const SessionDev* S = &v.sess[T.s];
        const LevelDev& Lv = S->lv[T.level];
        const int i = T.x0 + lx, j = T.y0 + ly;
        if (i >= Lv.cw || j >= Lv.ch) continue;
        float m[9];
        F3 o;
        ray_matrix(S, Lv, m, o);
        if (kFmt == KF_TSDF_F16U16 || (kFmt == kAnyFormat && S->fmt == KF_TSDF_F16U16))
            serial_ray<__half, MarchCount<kCount>, kBlocksPerSm == 3>(rq, S, T.s, m, o, T.level, i, j, budget, cnt);
        else
            serial_ray<float, MarchCount<kCount>, kBlocksPerSm == 3>(rq, S, T.s, m, o, T.level, i, j, budget, cnt);
    }
    cnt.flush(v.ray_counts);
}

template <class TF, class Cnt>
__device__ void coop_ray(const SessionDev* S, const LongRay& L, int lane, Cnt& cnt) {
    const TF* f = static_cast<const TF*>(S->tf);
    const RayGeo g = L.g;
    RayState st = L.st;
    float precise = 0.0f;
    march_coop(S, g, f, st, lane, precise, cnt);
    finish_ray_warp(S, g, f, L.level, L.i, L.j, precise, lane, st, cnt);
}

// The samples that a depth range left out at the end of a ray without a hit: it tells of the decisions in
// the ray's trace how many the march takes to the far plane.
__device__ __forceinline__ unsigned long long whole_trace(const SessionDev* S, RayState st, unsigned long long code) {
    const float large = S->mu * S->step_l;
    const int sw = int(code >> 40);
    if (sw) {   // small steps since sample sw - 1 of the large ones
        const float t = march_pos(st.base, sw - 1, large);
        st.base = (code >> 4 & 3) == 2 ? __fsub_rn(t, S->mu) : t;
        st.guard = sw - 1;
    }
    skip_to(st, st.far_d, sw ? S->mu * S->step_s : large);
    return (code & ~(0xffffffffull << 8)) | static_cast<unsigned long long>(st.guard) << 8;
}

// Debug mode, after the raycast: the traces of rays without a hit as if no depth range had ended them, so
// that they count what the march counts and 0 means a ray that never marched.
__global__ void __launch_bounds__(256) count_tails_kernel(EngineView v) {
    const int lane = threadIdx.x & 31, tw = v.tb->ray_tw;
    for (int t = blockIdx.x * 8 + (threadIdx.x >> 5); t < v.tb->n_ray; t += gridDim.x * 8) {
        const RayTile T = v.ray[t];
        const StepDev st = v.step[T.s];
        const SessionDev* S = &v.sess[T.s];
        const LevelDev& Lv = S->lv[T.level];
        const int i = T.x0 + lane % tw, j = T.y0 + lane / tw;
        if (!st.active || st.first || !S->range || !S->trace[T.level] || i >= Lv.cw || j >= Lv.ch) continue;
        unsigned long long* code = S->trace[T.level] + size_t(j) * Lv.w + i;
        if (*code & 3) continue;
        float m[9];
        F3 o;
        ray_matrix(S, Lv, m, o);
        RayGeo g;
        make_geo(S, m, o, i, j, g);
        RayState ray;
        if (ray_start(S, g, ray)) *code = whole_trace(S, ray, *code);
    }
}

// the queued long rays, one warp each
template <bool kCount>
__global__ void __launch_bounds__(256) raycast_long_kernel(EngineView v) {
    MarchCount<kCount> cnt;
    const int lane = threadIdx.x & 31;
    const int count = min(int(v.counters[6]), v.longq_cap);
    while (true) {
        int idx = 0;
        if (lane == 0) idx = int(atomicAdd(&v.counters[7], 1u));
        idx = __shfl_sync(0xffffffffu, idx, 0);
        if (idx >= count) break;
        const LongRay L = v.longq[idx];
        const SessionDev* S = &v.sess[L.s];
        if (S->fmt == KF_TSDF_F16U16)
            coop_ray<__half>(S, L, lane, cnt);
        else
            coop_ray<float>(S, L, lane, cnt);
    }
    cnt.flush(v.ray_counts);
}

int long_ray_bytes() { return int(sizeof(LongRay)); }

cudaError_t launch_ray_range(const EngineView& v, int grid, cudaStream_t st) {
    ray_range_kernel<<<grid, 256, 0, st>>>(v);
    return cudaGetLastError();
}

template <int kFmt>
static void launch_tiles(const EngineView& v, int grid, cudaStream_t st, bool many) {
    if (many) raycast_kernel<4, false, kFmt><<<grid, 256, 0, st>>>(v);
    else raycast_kernel<3, false, kFmt><<<grid, 256, 0, st>>>(v);
}

cudaError_t launch_raycast(const EngineView& v, int grid, int fmt, cudaStream_t st, bool many) {
    const bool count = v.ray_counts != nullptr;
    if (count) {
        if (many) raycast_kernel<4, true, kAnyFormat><<<grid, 256, 0, st>>>(v);
        else raycast_kernel<3, true, kAnyFormat><<<grid, 256, 0, st>>>(v);
    } else if (fmt == KF_TSDF_F32F32) {
        launch_tiles<KF_TSDF_F32F32>(v, grid, st, many);
    } else if (fmt == KF_TSDF_F16U16) {
        launch_tiles<KF_TSDF_F16U16>(v, grid, st, many);
    } else {
        launch_tiles<kAnyFormat>(v, grid, st, many);
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    if (count) raycast_long_kernel<true><<<grid, 256, 0, st>>>(v);
    else raycast_long_kernel<false><<<grid, 256, 0, st>>>(v);
    return cudaGetLastError();
}

int ray_count_slots() { return kRayCounts; }

cudaError_t launch_count_tails(const EngineView& v, cudaStream_t st) {
    count_tails_kernel<<<148 * 4, 256, 0, st>>>(v);
    return cudaGetLastError();
}

// ---- stage: kernel::raycast on a caller volume, and kf_render on a session's ----
//
// A caller's volume has no brick bounds, so the call makes them: one read of the distances of
// every block that the rays can reach, then the session's march -- 8 x 4-ray tiles, a lane budget,
// long rays by whole warps.  Bound by that read (HBM) and then by the march's instructions.  One
// thread per ray without skipping, as the reference marches, was bound by its longest rays (about
// 2,800 samples one after another): 640 x 480 rays in 512^3 f32 took 732 us in the kernel, now
// 168 in five (bounds 66, rays 58, long rays 31); kf_render's on a session's bounds 427 us, now 118.

struct RayStage {
    float m[9];      // R K^-1 (column-major)
    float o[3];
    float inv[9];    // its inverse: (p - o) to (pixel * t, t); valid when has_inv
    int has_inv;
};

// the scratch of one call, carved from one allocation
struct StageRayScratch {
    unsigned int* counters;   // [0] ray tiles, [1] long rays queued, [2] long rays taken
    unsigned int* range;      // directly after the counters: one memset clears both
    size_t clear_bytes;
    int* bmin;
    int* bdil;
    int* sdil;
    LongRay* longq;
    int longq_cap;
};

static size_t stage_ray_layout(int n, int w, int h, int longq_cap, char* base, StageRayScratch* s) {
    size_t at = 0;
    auto take = [&](size_t bytes) { const size_t o = at; at += (bytes + 255) & ~size_t(255); return base + o; };
    const size_t nb = size_t(n / 8), ns = (nb + 3) / 4;   // n = 0: no bounds
    StageRayScratch r;
    r.clear_bytes = (4 + size_t(range_words(w, h))) * sizeof(unsigned int);
    r.counters = reinterpret_cast<unsigned int*>(take(r.clear_bytes));
    r.range = r.counters + 4;
    r.bmin = reinterpret_cast<int*>(take(sizeof(int) * nb * nb * nb));
    r.bdil = reinterpret_cast<int*>(take(sizeof(int) * nb * nb * nb));
    r.sdil = reinterpret_cast<int*>(take(sizeof(int) * ns * ns * ns));
    r.longq = reinterpret_cast<LongRay*>(take(sizeof(LongRay) * size_t(longq_cap)));
    r.longq_cap = longq_cap;
    if (s) *s = r;
    return at;
}

size_t stage_raycast_scratch(int n, int w, int h, int longq_cap) {
    return stage_ray_layout(n, w, h, longq_cap, nullptr, nullptr);
}

__device__ __forceinline__ float min4(float4 v) { return fminf(fminf(v.x, v.y), fminf(v.z, v.w)); }
__device__ __forceinline__ float min_half2(unsigned int bits) {
    const float2 v = __half22float2(*reinterpret_cast<const __half2*>(&bits));
    return fminf(v.x, v.y);
}
__device__ __forceinline__ int order_key(float x) {   // order-preserving int of a float of either sign
    const int i = __float_as_int(x);
    return i >= 0 ? i : (i ^ 0x7fffffff);
}

// bmin of every 8^3 brick, one warp per 32 x 8 x 8 block.  A block that no ray of the image can
// sample -- its box, widened by the voxel that a sample's taps reach, lies outside one of the six
// planes of the rays' frustum -- is not read; its bound says 2, which no sample sees.  Else the
// warp reads 128-byte (f32) or 64-byte (f16) rows with all its 16-byte loads in flight.
template <class TF>
__global__ void __launch_bounds__(256) stage_bounds_kernel(const TF* f, int n, float vol_w, RayStage rs, int w, int h,
                                                           float min_d, float max_d, StageRayScratch s) {
    const int lane = threadIdx.x & 31, u = blockIdx.x * 8 + (threadIdx.x >> 5);
    const int ux = (n + 31) >> 5, uy = n >> 3, nb = n >> 3;
    if (u >= ux * uy * uy) return;
    const int x0 = (u % ux) * 32, y0 = ((u / ux) % uy) * 8, z0 = (u / (ux * uy)) * 8;
    int* out = s.bmin + (size_t(z0 >> 3) * nb + (y0 >> 3)) * nb + (x0 >> 3);
    const int bricks = min(4, nb - (x0 >> 3));
    if (rs.has_inv) {
        // lanes 0-7 (and their copies) hold the widened box's corners
        const float to_m = vol_w / float(n), mid = 0.5f * float(n) - 0.5f;
        const float px = ((lane & 1 ? float(min(x0 + 32, n)) + 0.05f : float(x0) - 1.05f) - mid) * to_m - rs.o[0];
        const float py = ((lane & 2 ? float(y0 + 8) + 0.05f : float(y0) - 1.05f) - mid) * to_m - rs.o[1];
        const float pz = ((lane & 4 ? float(z0 + 8) + 0.05f : float(z0) - 1.05f) - mid) * to_m - rs.o[2];
        const F3 q = mv3(rs.inv, F3{px, py, pz});   // (i t, j t, t); samples have i in [.5, w - .5]
        const unsigned int all = 0xffffffffu;
        if (__all_sync(all, q.x < 0.f) || __all_sync(all, q.x > float(w) * q.z) || __all_sync(all, q.y < 0.f) ||
            __all_sync(all, q.y > float(h) * q.z) || __all_sync(all, q.z < 0.999f * min_d) ||
            __all_sync(all, q.z > 1.001f * max_d)) {
            if (lane < bricks) out[lane] = 0x40000000;   // key of 2.0f
            return;
        }
    }
    float m = 3.0e38f;
    if constexpr (sizeof(TF) == 4) {
        const int x = x0 + 4 * (lane & 7);
        if (x < n) {
            const float4* p = reinterpret_cast<const float4*>(f + (size_t(z0) * n + y0 + (lane >> 3)) * n + x);
            const size_t row = size_t(n) / 4, slice = size_t(n) * row;   // n % 8 == 0
            float4 v[16];
#pragma unroll
            for (int k = 0; k < 16; ++k) v[k] = __ldg(p + (k >> 1) * slice + (k & 1) * 4 * row);
#pragma unroll
            for (int k = 0; k < 16; ++k) m = fminf(m, min4(v[k]));
        }
        m = fminf(m, __shfl_xor_sync(0xffffffffu, m, 1));
        m = fminf(m, __shfl_xor_sync(0xffffffffu, m, 8));
        m = fminf(m, __shfl_xor_sync(0xffffffffu, m, 16));
        if ((lane & 0x19) == 0 && x < n) out[lane >> 1] = order_key(m);
    } else {
        const int x = x0 + 8 * (lane & 3);
        if (x < n) {
            const uint4* p = reinterpret_cast<const uint4*>(f + (size_t(z0) * n + y0 + (lane >> 2)) * n + x);
            const size_t slice = size_t(n) * n / 8;
            uint4 v[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = __ldg(p + k * slice);
#pragma unroll
            for (int k = 0; k < 8; ++k)
                m = fminf(m, fminf(fminf(min_half2(v[k].x), min_half2(v[k].y)), fminf(min_half2(v[k].z), min_half2(v[k].w))));
        }
        m = fminf(m, __shfl_xor_sync(0xffffffffu, m, 4));
        m = fminf(m, __shfl_xor_sync(0xffffffffu, m, 8));
        m = fminf(m, __shfl_xor_sync(0xffffffffu, m, 16));
        if (lane < 4 && x < n) out[lane] = order_key(m);
    }
}

__global__ void __launch_bounds__(256) range_stage_kernel(const __grid_constant__ RangeView r, const int* bdil) {
    __shared__ unsigned short list[256 * 4];
    __shared__ int packed;
    const int tid = threadIdx.x, u0 = blockIdx.x * blockDim.x, ux = (r.n + 31) >> 5;
    const int count = block_pack(u0 + tid < fuse_units(r.n) ? range_candidates(r.n, r.nb, bdil, u0 + tid) : 0u, list, &packed);
    for (int i = tid & ~31; i < count; i += 256) {
        const bool on = i + (tid & 31) < count;
        const int code = on ? list[i + (tid & 31)] : 0, u = u0 + (code >> 2);
        range_bricks(r, on, (u % ux) * 4 + (code & 3), (u / ux) % r.nb, u / (ux * r.nb));
    }
}

// each warp pulls 8 x 4-ray tiles, as in a session's raycast
template <class TF>
__global__ void __launch_bounds__(256, 3) raycast_tiles_stage_kernel(const __grid_constant__ SessionDev S,
                                                                     const __grid_constant__ RayStage rs, int w, int h,
                                                                     int budget, StageRayScratch sc) {
    MarchCount<false> cnt;
    const int lane = threadIdx.x & 31, tx = (w + 7) / 8, ntiles = tx * ((h + 3) / 4);
    const RayQueue rq{sc.longq, sc.counters + 1, sc.longq_cap};
    while (true) {
        int t = 0;
        if (lane == 0) t = int(atomicAdd(sc.counters, 1u));
        t = __shfl_sync(0xffffffffu, t, 0);
        if (t >= ntiles) break;
        const int i = (t % tx) * 8 + (lane & 7), j = (t / tx) * 4 + (lane >> 3);
        if (i >= w || j >= h) continue;
        serial_ray<TF, MarchCount<false>, true>(rq, &S, 0, rs.m, F3{rs.o[0], rs.o[1], rs.o[2]}, 0, i, j, budget, cnt);
    }
}

template <class TF>
__global__ void __launch_bounds__(256) raycast_long_stage_kernel(const __grid_constant__ SessionDev S, StageRayScratch sc) {
    MarchCount<false> cnt;
    const int lane = threadIdx.x & 31;
    const int count = min(int(sc.counters[1]), sc.longq_cap);
    while (true) {
        int idx = 0;
        if (lane == 0) idx = int(atomicAdd(sc.counters + 2, 1u));
        idx = __shfl_sync(0xffffffffu, idx, 0);
        if (idx >= count) break;
        coop_ray<TF>(&S, sc.longq[idx], lane, cnt);
    }
}

// one thread per ray, no scratch: for a call under stream capture, or one that finds no memory
template <class TF>
__global__ void raycast_stage_kernel(SessionDev S, RayStage rs, int w, int h) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= w || j >= h) return;
    const TF* f = static_cast<const TF*>(S.tf);
    RayGeo g;
    make_geo(&S, rs.m, F3{rs.o[0], rs.o[1], rs.o[2]}, i, j, g);
    RayState st;
    if (!ray_start(&S, g, st)) {
        write_miss(&S, 0, i, j);
        return;
    }
    float precise = 0.0f;
    MarchCount<false> cnt;
    march_serial<TF, MarchCount<false>, false>(&S, g, f, st, 0x7fffffff, precise, cnt);
    finish_ray(&S, g, f, 0, i, j, precise, st, cnt);
}

// Bounds cost a read of the visible volume whatever the image, and the march without them costs in
// proportion to the rays, in volumes of every size (a finer volume has more samples per ray).  Both
// ways measured with cold caches, us, without / with bounds, in 64^3, 128^3, 256^3 and 512^3 f32:
//   320x240   44 / 48    60 / 58    79 / 89   130 / 179
//   400x300   44 / 48    63 / 62    81 / 91   142 / 175
//   480x360   48 / 52    73 / 71    93 / 93   183 / 181
//   640x480   57 / 62    99 / 87   121 / 101  245 / 181
// (512^3 f16: 400x300 137 / 141, 480x360 180 / 146.)  The line lies between the middle two images; in
// 64^3 it costs 4 us, in 128^3 it gives away 2.
constexpr long long kBoundsRays = 160000;

// A depth range that begins behind the camera has no bounds: the frustum's planes and the depth ranges
// hold for samples ahead of it.
bool stage_raycast_builds_bounds(const kf_volume* vol, int w, int h, float min_d) {
    return min_d >= 0.0f && (long long)w * h >= kBoundsRays &&
           reinterpret_cast<uintptr_t>(vol->f) % 16 == 0;   // vector reads
}

// Without bounds a lane's budget is short for small images, whose few warps leave the GPU idle
// while a lane marches (512^3 f32, cold caches: 80x60 76 us at 24, 106 at 64, 160x120 90 and 111), and
// long enough to reach most surfaces for larger ones (320x240 165 and 130, 400x300 222 and 142; in 128^3,
// whose rays are short, 44 and 60, 52 and 63).
static int budget_without_bounds(int w, int h) { return (long long)w * h <= 24000 ? 24 : 64; }

// Every ray of a march without bounds may outlast its budget, and a ray that finds the queue full
// marches on alone, several times slower; with bounds few do (long_ray_entries).
int stage_raycast_queue(int w, int h, bool bounds, long long share) {
    const long long rays = (long long)w * h;
    return int(bounds ? share : std::max(share, std::min(rays, 1LL << 18)));
}

template <class TF>
static cudaError_t launch_stage(SessionDev& S, const RayStage& rs, int w, int h, bool build, void* scratch,
                                int longq_cap, cudaStream_t st) {
    if (!scratch) {
        const dim3 blk(8, 8), grd((w + 7) / 8, (h + 7) / 8);
        raycast_stage_kernel<TF><<<grd, blk, 0, st>>>(S, rs, w, h);
        return cudaGetLastError();
    }
    StageRayScratch sc;
    stage_ray_layout(build ? S.n : 0, w, h, longq_cap, static_cast<char*>(scratch), &sc);
    cudaError_t e = cudaMemsetAsync(sc.counters, 0, sc.clear_bytes, st);
    if (e != cudaSuccess) return e;
    if (build) {
        S.nb = S.n / 8;
        S.ns = (S.nb + 3) / 4;
        S.bdil = sc.bdil;
        S.sdil = sc.sdil;
        stage_bounds_kernel<TF><<<(fuse_units(S.n) + 7) / 8, 256, 0, st>>>(static_cast<const TF*>(S.tf), S.n, S.vol_w, rs,
                                                                           w, h, S.min_d, S.max_d, sc);
        e = launch_widen_bricks(sc.bmin, sc.bdil, sc.sdil, S.n, st);
        if (e != cudaSuccess) return e;
    }
    if (S.bdil && rs.has_inv && S.n >= kRangeMinN) {
        S.range = sc.range;
        S.rgw = (w + kRangeTile - 1) / kRangeTile;
        S.rgh = (h + kRangeTile - 1) / kRangeTile;
        RangeView r;
        for (int q = 0; q < 9; ++q) r.P[q] = rs.inv[q];
        for (int q = 0; q < 3; ++q) r.o[q] = rs.o[q];
        r.w = w; r.h = h; r.rgw = S.rgw; r.rgh = S.rgh;
        r.min_d = S.min_d; r.max_d = S.max_d; r.vol_w = S.vol_w;
        r.n = S.n; r.nb = S.nb;
        r.range = sc.range;
        range_stage_kernel<<<(fuse_units(S.n) + 255) / 256, 256, 0, st>>>(r, S.bdil);
    }
    const int tiles = ((w + 7) / 8) * ((h + 3) / 4), grid = std::min(148 * 6, (tiles + 7) / 8);
    raycast_tiles_stage_kernel<TF><<<grid, 256, 0, st>>>(S, rs, w, h, S.bdil ? kSerialBudgetSingle : budget_without_bounds(w, h), sc);
    raycast_long_stage_kernel<TF><<<148 * 4, 256, 0, st>>>(S, sc);
    return cudaGetLastError();
}

cudaError_t stage_raycast(const kf_volume* vol, const float* pose, const float* ik, float4* vtx, float4* nrm, int w,
                          int h, float min_d, float max_d, float step_l, float step_s, void* scratch, int longq_cap,
                          cudaStream_t st, const SessionDev* bounds) {
    SessionDev S{};
    if (bounds) {   // a session's brick bounds: the same samples, skipping exactly as the pipeline
        S.bdil = bounds->bdil;
        S.sdil = bounds->sdil;
        S.nb = bounds->nb;
        S.ns = bounds->ns;
    }
    S.n = vol->n;
    S.fmt = vol->format;
    S.vol_w = vol->width;
    S.mu = vol->mu;
    S.tf = vol->f;
    S.tw = vol->w;
    S.min_d = min_d;
    S.max_d = max_d;
    S.step_l = step_l;
    S.step_s = step_s;
    S.keep_on_miss = 1;
    S.pv[0] = vtx;
    S.pn[0] = nrm;
    S.lv[0].w = w;
    S.lv[0].h = h;
    S.lv[0].cw = w;
    S.lv[0].ch = h;
    RayStage rs;
    // R * K^-1 with every product and sum rounded on its own (ray_matrix's arithmetic)
    for (int col = 0; col < 3; ++col)
        for (int row = 0; row < 3; ++row) {
            const volatile float a = pose[row] * ik[col * 3 + 0], b = pose[4 + row] * ik[col * 3 + 1],
                                 c = pose[8 + row] * ik[col * 3 + 2];
            const volatile float ab = a + b;
            rs.m[col * 3 + row] = ab + c;
        }
    rs.o[0] = pose[12];
    rs.o[1] = pose[13];
    rs.o[2] = pose[14];
    // the inverse (adjugate over determinant), only to place the frustum's planes
    {
        const float* m = rs.m;
        const double a = m[0], b = m[3], c = m[6], d = m[1], e = m[4], f = m[7], g = m[2], hh = m[5], i = m[8];
        const double det = a * (e * i - f * hh) - b * (d * i - f * g) + c * (d * hh - e * g);
        const double adj[9] = {e * i - f * hh, f * g - d * i, d * hh - e * g, c * hh - b * i, a * i - c * g,
                               b * g - a * hh, b * f - c * e, c * d - a * f, a * e - b * d};
        rs.has_inv = 1;
        for (int q = 0; q < 9; ++q) {
            rs.inv[q] = float(adj[q] / det);
            if (!std::isfinite(rs.inv[q])) rs.has_inv = 0;
        }
    }
    const bool build = !bounds && stage_raycast_builds_bounds(vol, w, h, min_d);
    if (vol->format == KF_TSDF_F16U16) return launch_stage<__half>(S, rs, w, h, build, scratch, longq_cap, st);
    return launch_stage<float>(S, rs, w, h, build, scratch, longq_cap, st);
}

}  // namespace kf
