// k_tsdf.cu -- TSDF volume: initialisation, projective fusion, brick bounds, layout conversion.
//
// Reference: initializeGridKernel (project/src/tsdf.cu:7-18) and fuseKernel
// (project/src/tsdf.cu:20-75), which walks one (x, y) voxel column per thread through a
// cudaArray surface with 4-byte reads and writes, projecting every voxel of the volume.
//
// Here the volume is two linear arrays in HBM (distance, weight; x fastest), cut into units of
// 32 x 8 x 8 voxels and their 16 x 8 x 8 halves.  Two launches per frame:
//   - fuse_cull_kernel tests every unit of every session as a whole, one unit per thread, from its 8
//     projected corners (the projection of a box in front of the camera lies inside its corners'
//     bounding box): outside the depth range or the image, no valid depth under it, or every voxel
//     more than mu behind the farthest valid depth under it -- then no voxel of it can update.  The
//     halves of the units that pass are tested the same way, and the survivors (a few percent of a
//     512^3 volume) are appended to a queue with one atomic per warp.
//   - fuse_kernel's persistent warps walk the queued halves row by row, eight slices at a time, each
//     lane four consecutive voxels along x, which it reads and writes as 16-byte (f32) or 8-byte (f16)
//     vectors.
// What bounds the second is the L1's data pipe, which serves a request one 128-byte line at a time, and
// after it instruction issue.  Whole units (32 x 2 x 2 voxels a step, 42 % of them updating) took 50 us
// for one 640x480 frame into 512^3 f32 and 824 us for 24 into 512^3 f16+u16; 8^3 bricks, which fit the
// surface best but put every access on 16 lines, 39 and 671; halves with their slices across the lanes
// (8 lines an access, and gathers that fall on two or three image rows) 30 and 530.
// Each 8^3 brick keeps a lower bound of its distances (an atomic minimum: values that fusion stores
// below one of the raycast's two thresholds lower it to one of two levels), widened to the 2 x 2 x 2
// bricks a trilinear sample can touch and to 32^3 super-bricks; fusion lowers the widened bounds itself
// whenever a brick's bound falls, so no pass recomputes them.  The raycaster skips samples whose bound proves they cannot matter.
#include "kf_host.h"

namespace kf {

// order-preserving int key of a float (atomicMin on floats of either sign)
__device__ __forceinline__ int fkey(float x) {
    const int i = __float_as_int(x);
    return i >= 0 ? i : (i ^ 0x7fffffff);
}

// A brick's lower bound may have fallen to key k: the widened bounds of every brick and super-brick whose
// neighbourhood holds the brick fall with it -- bdil of bricks b - {0,1}^3 (a brick's bdil
// covers {b, b+1}^3) and sdil of super-bricks s with 4 s <= b <= 4 s + 4 per axis.  Bounds only
// ever fall (atomic minima), so these running minima are exactly the minima over each
// neighbourhood.  Most calls find the bound already at or below k.
// `seen`: a value the bound had earlier (a stale value is never below it).
__device__ __forceinline__ void lower_brick_bound(const FuseCtx& c, int bx, int by, int bz, int k, int seen) {
    const int nb = c.nb;
    int* pb = c.bmin + (size_t(bz) * nb + by) * nb + bx;
    if (k >= seen) return;
    if (k >= atomicMin(pb, k)) return;    // another warp lowered it as far already
#pragma unroll
    for (int d = 0; d < 8; ++d) {
        const int x = bx - (d & 1), y = by - ((d >> 1) & 1), z = bz - (d >> 2);
        if (x >= 0 && y >= 0 && z >= 0) atomicMin(c.bdil + (size_t(z) * nb + y) * nb + x, k);
    }
    const int ns = c.ns;
#pragma unroll
    for (int d = 0; d < 8; ++d) {
        // super-brick b / 4 per axis, and b / 4 - 1 when b is the last brick of its range too
        const int x = (bx >> 2) - (d & 1), y = (by >> 2) - ((d >> 1) & 1), z = (bz >> 2) - (d >> 2);
        const bool ok = ((d & 1) == 0 || ((bx & 3) == 0 && bx > 0)) && (((d >> 1) & 1) == 0 || ((by & 3) == 0 && by > 0)) &&
                        ((d >> 2) == 0 || ((bz & 3) == 0 && bz > 0));
        if (ok && x < ns && y < ns && z < ns) atomicMin(c.sdil + (size_t(z) * ns + y) * ns + x, k);
    }
}

// The approximate reciprocal.  a * rcp_approx(b) has the bits of __fdividef(a, b) for every b that is
// not denormal (compared over 4 M pairs); depths above kMinDepth and sums with their reciprocals are none.
__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// running weighted average (project/src/tsdf.cu:56-69, built with -use_fast_math: the
// division is the approximate one); max_w > 0 clamps the weight
__device__ __forceinline__ void fuse_update(float& F, float& Wt, float fn, float wn, float max_w) {
    F = __fmul_rn(__fmaf_rn(F, Wt, __fmul_rn(fn, wn)), rcp_approx(__fadd_rn(Wt, wn)));
    float w1 = __fadd_rn(Wt, wn);
    if (max_w > 0.0f) w1 = fminf(w1, max_w);
    Wt = w1;
}

// true when no voxel of the block [x0, x0+nx) x [j0, j0+8) x [k0, k0+8) can update; one
// thread tests one block
__device__ __forceinline__ bool block_culled(const FuseCtx& c, int x0, int nx, int j0, int k0) {
    const int n = c.n;
    const float xa = __ldg(c.xs + x0), xb = __ldg(c.xs + min(x0 + nx - 1, n - 1));
    const float ya = __ldg(c.xs + j0), yb = __ldg(c.xs + min(j0 + 7, n - 1));
    const float za = __ldg(c.zs + k0), zb = __ldg(c.zs + min(k0 + 7, n - 1));
    float ex[8], ey[8], ez[8];
    float zmin = 3.0e38f, zmax = -3.0e38f;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const float x = (q & 1) ? xb : xa, y = (q & 2) ? yb : ya, z = (q & 4) ? zb : za;
        // same operation order as the per-voxel projection below
        const float bx = c.iR[3] * y + c.iR[6] * z + c.it[0];
        const float by = c.iR[4] * y + c.iR[7] * z + c.it[1];
        const float bz = c.iR[5] * y + c.iR[8] * z + c.it[2];
        ex[q] = c.iR[0] * x + bx;
        ey[q] = c.iR[1] * x + by;
        ez[q] = c.iR[2] * x + bz;
        zmin = fminf(zmin, ez[q]);
        zmax = fmaxf(zmax, ez[q]);
    }
    if (zmax < c.min_d - 1e-4f || zmin >= c.max_d + 1e-4f) return true;
    if (!(zmin > 1e-3f)) return false;   // a corner behind the camera: no image bound
    float pxmin = 3.0e38f, pxmax = -3.0e38f, pymin = 3.0e38f, pymax = -3.0e38f;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        // approximate division (a few 1e-4 px at most): the bounds below keep 0.01 px margins
        const float iz = rcp_approx(ez[q]);
        const float px = (c.fx * ex[q] + c.cx * ez[q]) * iz;
        const float py = (c.fy * ey[q] + c.cy * ez[q]) * iz;
        pxmin = fminf(pxmin, px);
        pxmax = fmaxf(pxmax, px);
        pymin = fminf(pymin, py);
        pymax = fmaxf(pymax, py);
    }
    if (pxmax < -0.01f || pxmin > float(c.w) + 0.01f || pymax < -0.01f || pymin > float(c.h) + 0.01f) return true;
    if (!c.dmax) return false;
    const int tx0 = min(max(int(pxmin - 0.01f), 0), c.w - 1) >> 4;
    const int tx1 = min(max(int(pxmax + 0.01f), 0), c.w - 1) >> 4;
    const int ty0 = min(max(int(pymin - 0.01f), 0), c.h - 1) >> 4;
    const int ty1 = min(max(int(pymax + 0.01f), 0), c.h - 1) >> 4;
    // A box over many tiles is near the camera or coarse, and seldom behind every depth under it; one
    // thread reading them all held the launch (frame and visualization volume of 256^3 over 8 m and
    // 512^3 over 5 m, cull + cull: 28 + 13 us with up to 512 tiles, 12 + 11 with 32, 11 + 10 with 8, where
    // fusion takes 10 us more; 512^3 over 3 m the same with 32 and 512).
    if ((tx1 - tx0 + 1) * (ty1 - ty0 + 1) > 32) return false;
    float dm = 0.0f;
    for (int ty = ty0; ty <= ty1; ++ty)
        for (int tx = tx0; tx <= tx1; ++tx) dm = fmaxf(dm, __ldg(c.dmax + size_t(ty) * c.t16w + tx));
    // every voxel meets either an invalid depth or d - z <= dm - zmin < -mu (the margin also covers
    // the sum's rounding where depths are in the thousands: a caller's maps in millimetres)
    return dm == 0.0f || zmin > dm + c.mu + 1e-4f + 1e-6f * dm;
}

// block coordinates of fusion unit u of an n^3 volume (units: 32 x 8 x 8 blocks, x fastest)
__device__ __forceinline__ void unit_origin(int n, int u, int& x0, int& j0, int& k0) {
    const int ux = (n + 31) >> 5, uy = (n + 7) >> 3;
    x0 = (u % ux) * 32;
    j0 = ((u / ux) % uy) * 8;
    k0 = (u / (ux * uy)) * 8;
}

// four consecutive voxels of a row as one vector: 16 bytes of f32, 8 bytes of f16 or u16
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ uint2 ld4(const __half* p) { return *reinterpret_cast<const uint2*>(p); }
__device__ __forceinline__ uint2 ld4(const uint16_t* p) { return *reinterpret_cast<const uint2*>(p); }
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void st4(__half* p, uint2 v) { *reinterpret_cast<uint2*>(p) = v; }
__device__ __forceinline__ void st4(uint16_t* p, uint2 v) { *reinterpret_cast<uint2*>(p) = v; }
// component q of a 4-vector (q a compile-time constant after unrolling)
__device__ __forceinline__ float& comp(float4& v, int q) { return q == 0 ? v.x : q == 1 ? v.y : q == 2 ? v.z : v.w; }

// fuseKernel (project/src/tsdf.cu:28-74) for the 16 x 8 x 8 half of a unit at (x0, j0, k0), one warp.
// Lane l takes four consecutive voxels along x, 4 (l & 3), of slice k0 + (l >> 2), and step s row
// y = j0 + s: 128 voxels a step, each lane a vector read-modify-write of 16 (f32) or 8 (f16, u16)
// bytes.  The warp takes steps [s0, s1).  The slices go across the lanes because a row's pixels hardly
// move with depth: a step's gathers fall on two or three image rows, where eight rows of a slice would
// fall on eight.  A vector whose voxels all stay unchanged is not written; voxels that stay unchanged
// inside a written vector are written back with their own bits.
template <class TF, class TW>
__device__ __forceinline__ void fuse_half(const FuseCtx& c, int x0, int j0, int k0, int s0, int s1, int lane) {
    const int n = c.n;
    const int x = x0 + 4 * (lane & 3), k = k0 + (lane >> 2);
    const bool lane_in = x < n;   // n % 8 == 0: all four voxels or none
    // what each voxel needs of the context in registers, the rest read once per step
    const float r0 = c.iR[0], r1 = c.iR[1], r2 = c.iR[2];
    const float fx = c.fx, fy = c.fy, cx = c.cx, cy = c.cy, min_d = c.min_d, max_d = c.max_d, mu = c.mu, max_w = c.max_w;
    const unsigned int w = unsigned(c.w), h = unsigned(c.h);
    const float4 xv = lane_in ? __ldg(reinterpret_cast<const float4*>(c.xs + x)) : make_float4(0.f, 0.f, 0.f, 0.f);
    const float z = __ldg(c.zs + k);
    const float z0 = __fmul_rn(c.iR[6], z), z1 = __fmul_rn(c.iR[7], z), z2 = __fmul_rn(c.iR[8], z);
    const float inv_mu = rcp_approx(mu);
    size_t at = (size_t(k) * n + j0 + s0) * n + x;
    float kmin = 3.0e38f;   // the smallest distance this lane stores
    // the bounds of the half unit's two bricks, lanes 0 and 2: read ahead of their use
    const bool bounds = c.bmin && (lane & ~2) == 0 && lane_in;
    const int seen = bounds ? __ldcg(c.bmin + (size_t(k0 >> 3) * c.nb + (j0 >> 3)) * c.nb + (x >> 3)) : 0;
#pragma unroll 1
    for (int j = j0 + s0; j < j0 + s1; ++j, at += n) {
        const float y = __ldg(c.xs + j);
        const float bx = __fadd_rn(__fmaf_rn(c.iR[3], y, z0), c.it[0]);
        const float by = __fadd_rn(__fmaf_rn(c.iR[4], y, z1), c.it[1]);
        const float bz = __fadd_rn(__fmaf_rn(c.iR[5], y, z2), c.it[2]);
        float pz[4], d[4];
        unsigned int upd = 0;
        // project, and gather the nearest pixels' depths
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float xq = q == 0 ? xv.x : q == 1 ? xv.y : q == 2 ? xv.z : xv.w;
            const float ex = __fmaf_rn(r0, xq, bx), ey = __fmaf_rn(r1, xq, by), ez = __fmaf_rn(r2, xq, bz);
            // pixel /= pixel.z: the reference's build divides approximately, but rounded
            // division here keeps the per-frame pose within 2e-6 rad of the FP64 oracle
            // (1e-4 with the approximate one: voxels near a pixel edge change pixel)
            const float iz = 1.0f / ez;
            const float px = __fmul_rn(__fmaf_rn(fx, ex, __fmul_rn(cx, ez)), iz);
            const float py = __fmul_rn(__fmaf_rn(fy, ey, __fmul_rn(cy, ez)), iz);
            // floor as the low bits of p + 2^23 rounded down: exact for 0 <= p < 2^23, and any other
            // value (negative, larger, not a number) leaves an integer no image reaches
            const unsigned int ix = __float_as_uint(__fadd_rd(px, 8388608.0f)) - 0x4B000000u;
            const unsigned int iy = __float_as_uint(__fadd_rd(py, 8388608.0f)) - 0x4B000000u;
            const bool in = lane_in && ez >= min_d && ez < max_d && ix < w && iy < h;
            pz[q] = ez;
            d[q] = in ? __ldg(c.depth + (iy * w + ix)) : 0.0f;   // 0: no valid depth
        }
        float fn[4], wn[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float diff = d[q] - pz[q];
            // the reference divides with -use_fast_math: diff times the approximate 1 / mu
            fn[q] = fminf(1.0f, __fmul_rn(diff, inv_mu));
            wn[q] = rcp_approx(d[q]);   // its 1 / depth is the fast reciprocal too
            if (depth_valid(d[q]) && diff >= -mu) upd |= 1u << q;
        }
        if (!upd) continue;
        TF* const F = static_cast<TF*>(c.F) + at;
        TW* const Wa = static_cast<TW*>(c.W) + at;
        auto fv = ld4(F);
        auto wv = ld4(Wa);
        // one vector read-modify-write of the lane's four voxels
        if constexpr (sizeof(TF) == 4) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                float f0 = comp(fv, q), w0 = comp(wv, q);
                fuse_update(f0, w0, fn[q], wn[q], max_w);
                if (upd & (1u << q)) {
                    comp(fv, q) = f0;
                    comp(wv, q) = w0;
                    kmin = fminf(kmin, f0);
                }
            }
            st4(F, fv);
            st4(Wa, wv);
        } else {
            // All four voxels are decoded and encoded again, the unchanged ones exactly: an fp16
            // value survives float and back, and a weight u / 1024 survives the scaling by a
            // power of two.  The weight steps u < 2^16 become floats as the float 2^23 + u
            // (bits 0x4B000000 | u) less 2^23, and return as the low bits of x + 2^23, whose
            // round-to-nearest-even addition is rintf(x) for 0 <= x < 2^22: exact, without
            // conversion instructions.
            static_assert(KF_WEIGHT_SCALE == 1024.0f, "weights are steps of 1 / 1024");
            const float2 f01 = __half22float2(*reinterpret_cast<const __half2*>(&fv.x));
            const float2 f23 = __half22float2(*reinterpret_cast<const __half2*>(&fv.y));
            float f[4] = {f01.x, f01.y, f23.x, f23.y}, wt[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const unsigned int bits = __byte_perm(q < 2 ? wv.x : wv.y, 0x4B000000u, (q & 1) ? 0x7632 : 0x7610);
                wt[q] = __fmul_rn(__fsub_rn(__uint_as_float(bits), 8388608.0f), 1.0f / KF_WEIGHT_SCALE);
                if (upd & (1u << q)) fuse_update(f[q], wt[q], fn[q], wn[q], max_w);
            }
            const __half2 h01 = __floats2half2_rn(f[0], f[1]), h23 = __floats2half2_rn(f[2], f[3]);
            fv.x = *reinterpret_cast<const unsigned int*>(&h01);
            fv.y = *reinterpret_cast<const unsigned int*>(&h23);
            unsigned int wb[4];
#pragma unroll
            for (int q = 0; q < 4; ++q)
                wb[q] = __float_as_uint(__fadd_rn(fminf(__fmul_rn(wt[q], KF_WEIGHT_SCALE), 65535.0f), 8388608.0f));
            wv.x = __byte_perm(wb[0], wb[1], 0x5410);
            wv.y = __byte_perm(wb[2], wb[3], 0x5410);
            const float2 r01 = __half22float2(h01), r23 = __half22float2(h23);
            const float r[4] = {r01.x, r01.y, r23.x, r23.y};
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (upd & (1u << q)) kmin = fminf(kmin, r[q]);
            st4(F, fv);
            st4(Wa, wv);
        }
    }
    if (c.bmin) {
        // The raycast asks of a bound only on which side of its two thresholds it lies, so a bound
        // falls to one of two values: free space whose running average creeps below 1 by roundings
        // then changes no bound, nor does a surface's noise.
        const unsigned int low = __ballot_sync(0xffffffffu, kmin < kSkipLarge);
        if (low == 0) return;
        const unsigned int solid = __ballot_sync(0xffffffffu, kmin < kSkipSmall);
        const unsigned int brick = lane & 2 ? 0xccccccccu : 0x33333333u;   // the lanes of this lane's brick
        if (bounds && (low & brick))
            lower_brick_bound(c, x >> 3, j0 >> 3, k0 >> 3, fkey(solid & brick ? -1.0f : kSkipSmall), seen);
    }
}

// part `part` of `split` (1, 2 or 4) of packed half unit b
template <int kFmt>
__device__ __forceinline__ void fuse_part(const FuseCtx& c, unsigned int b, unsigned int part, unsigned int split, int lane) {
    const int x0 = int(b & 1023u) * 8, j0 = int(b >> 10 & 1023u) * 8, k0 = int(b >> 20) * 8;
    const int steps = int(8u / split), s0 = int(part) * steps;
    if (kFmt == KF_TSDF_F16U16 || (kFmt == kAnyFormat && c.fmt == KF_TSDF_F16U16))
        fuse_half<__half, uint16_t>(c, x0, j0, k0, s0, s0 + steps, lane);
    else
        fuse_half<float, float>(c, x0, j0, k0, s0, s0 + steps, lane);
}

FuseCtx fuse_context(const SessionDev& d, bool vis) {
    FuseCtx c{};
    c.fx = d.lv[0].fx; c.fy = d.lv[0].fy; c.cx = d.lv[0].cx; c.cy = d.lv[0].cy;
    c.min_d = d.min_d; c.max_d = d.max_d; c.max_w = d.max_w;
    c.depth = d.depth_m;
    c.dmax = d.dmax16;
    c.t16w = d.t16w;
    c.w = d.W; c.h = d.H; c.fmt = d.fmt;
    if (vis) {
        const VisDev& V = d.vis;
        c.mu = V.mu; c.n = V.n; c.nb = V.nb; c.ns = V.ns;
        c.F = V.tf; c.W = V.tw; c.xs = V.xs; c.zs = V.zs; c.bmin = V.bmin; c.bdil = V.bdil; c.sdil = V.sdil;
    } else {
        c.mu = d.mu; c.n = d.n; c.nb = d.nb; c.ns = d.ns;
        c.F = d.tf; c.W = d.tw; c.xs = d.xs; c.zs = d.zs; c.bmin = d.bmin; c.bdil = d.bdil; c.sdil = d.sdil;
    }
    return c;
}

// a warp copies a context to shared memory
__device__ __forceinline__ void load_ctx(const FuseCtx* from, FuseCtx& c, int lane) {
    static_assert(sizeof(FuseCtx) % 16 == 0 && sizeof(FuseCtx) <= 32 * 16, "one vector per lane");
    if (lane < int(sizeof(FuseCtx) / 16)) reinterpret_cast<uint4*>(&c)[lane] = __ldcg(reinterpret_cast<const uint4*>(from) + lane);
}

// which tables a fusion launch walks: the tracking volumes' or the visualization volumes'
template <bool kVis> struct FuseLists;
template <> struct FuseLists<false> {
    static __device__ long long total(const EngineView& v) { return v.tb->fuse_total; }
    static __device__ const FuseCtx* ctx(const EngineView& v) { return v.fctx; }
    static __device__ const long long* prefix(const EngineView& v) { return v.fuse_prefix; }
    static __device__ uint2* queue(const EngineView& v) { return v.fuseq; }
    static __device__ int queue_cap(const EngineView& v) { return v.fuseq_cap; }
    static constexpr int kQueued = 4, kTaken = 5;   // counters
};
template <> struct FuseLists<true> {
    static __device__ long long total(const EngineView& v) { return v.tb->vis_fuse_total; }
    static __device__ const FuseCtx* ctx(const EngineView& v) { return v.vis_fctx; }
    static __device__ const long long* prefix(const EngineView& v) { return v.vis_fuse_prefix; }
    static __device__ uint2* queue(const EngineView& v) { return v.vis_fuseq; }
    static __device__ int queue_cap(const EngineView& v) { return v.vis_fuseq_cap; }
    static constexpr int kQueued = 8, kTaken = 9;
};

// a queue entry: the session and the half unit's first brick (n <= 8192: ten bits per coordinate)
__device__ __forceinline__ unsigned int pack_brick(int bx, int by, int bz) {
    return unsigned(bx) | unsigned(by) << 10 | unsigned(bz) << 20;
}

// the 16-voxel halves that exist of the unit at x0
__device__ __forceinline__ unsigned int unit_halves(int n, int x0) { return n - x0 > 16 ? 3u : 1u; }

// Two tests per block of threads: one thread per 32 x 8 x 8 unit of every stepping session, then one
// per 16 x 8 x 8 half of the units that passed (packed), whose box shares fewer pixels and depths.  The
// halves that can update are appended to the queue (counters[4] = entries; [8] for the visualization
// volumes), one atomic per warp.
template <bool kVis>
__global__ void __launch_bounds__(256, 4) fuse_cull_kernel(EngineView v) {
    using Lists = FuseLists<kVis>;
    __shared__ unsigned short list[256 * 4];
    __shared__ int packed;
    const long long total = Lists::total(v);
    const long long* prefix = Lists::prefix(v);
    uint2* queue = Lists::queue(v);
    const int queue_cap = Lists::queue_cap(v);
    const int S_cap = v.tb->S;
    const int tid = threadIdx.x, lane = tid & 31;
    const long long stride = (long long)gridDim.x * blockDim.x;
    if (!kVis) {
        // the raycast of this step is done with the sessions' depth ranges: zero for the next one
        for (int s = blockIdx.x; s < S_cap; s += gridDim.x) {
            const SessionDev* S = &v.sess[s];
            if (!v.step[s].active || !S->range) continue;
            for (int q = tid; q < range_words(S->W, S->H); q += blockDim.x) S->range[q] = 0u;
        }
    }
    FuseCtx c;
    int cur_s = -1;
    bool live = false;
    auto enter = [&](int s) {
        if (s == cur_s) return;
        cur_s = s;
        c = Lists::ctx(v)[s];
        live = v.step[s].active && c.ok;
    };
    for (long long base = (long long)blockIdx.x * blockDim.x; base < total; base += stride) {
        unsigned int m = 0;
        if (base + tid < total) {
            const int s = unit_session(prefix, base + tid, S_cap);
            enter(s);
            if (live) {
                int x0, j0, k0;
                unit_origin(c.n, int(base + tid - __ldg(prefix + s)), x0, j0, k0);
                if (!block_culled(c, x0, 32, j0, k0)) m = unit_halves(c.n, x0);
            }
        }
        const int count = block_pack(m, list, &packed);
        for (int i = tid & ~31; i < count; i += 256) {
            bool keep = false;
            uint2 entry = make_uint2(0u, 0u);
            if (i + lane < count) {
                const int code = list[i + lane];
                const long long g = base + (code >> 2);
                const int s = unit_session(prefix, g, S_cap);
                enter(s);   // live: its unit passed
                int x0, j0, k0;
                unit_origin(c.n, int(g - __ldg(prefix + s)), x0, j0, k0);
                keep = !block_culled(c, x0 + 16 * (code & 3), 16, j0, k0);
                entry = make_uint2(unsigned(s), pack_brick((x0 >> 3) + 2 * (code & 3), j0 >> 3, k0 >> 3));
            }
            const unsigned int km = __ballot_sync(0xffffffffu, keep);
            if (km == 0) continue;
            unsigned int slot = 0;
            if (lane == 0) slot = atomicAdd(&v.counters[Lists::kQueued], unsigned(__popc(km)));
            slot = __shfl_sync(0xffffffffu, slot, 0);
            const unsigned int at = slot + __popc(km & ((1u << lane) - 1u));
            if (keep && at < unsigned(queue_cap)) queue[at] = entry;   // capacity >= all halves
        }
        __syncthreads();   // the list and its count are read before the next units' are written
    }
}

constexpr int kFuseWarps = 8;

// How many warps share a half unit: four while the queue holds no more than one per warp (small
// volumes: the steps of a half unit are a chain of round trips), two up to four per warp (a single
// session's frame), else one.  Which warp fuses which rows changes no voxel's arithmetic.
__device__ __forceinline__ unsigned int fuse_split(unsigned int halves, unsigned int warps) {
    return halves <= warps ? 4u : halves <= 4u * warps ? 2u : 1u;
}

// Persistent warps.  Items (half units, or their halves or quarters) go to the warps in turn while
// there are few, and beyond kStaticItems per warp in runs from a counter: atomics on one address
// complete one in about 0.7 ns, whichever SM they come from, so a counter asked for every item costs
// a kernel of short items its time (one session's 16 thousand items: 37 us with it, 30 without).  The next item's queue
// entry is read while an item is fused.
constexpr unsigned int kStaticItems = 16;

template <bool kVis, int kFmt>
__global__ void __launch_bounds__(256, 4) fuse_kernel(EngineView v) {
    using Lists = FuseLists<kVis>;
    __shared__ FuseCtx ctx[kFuseWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint2* queue = Lists::queue(v);
    unsigned int* const taken = &v.counters[Lists::kTaken];
    const unsigned int halves = min(__ldcg(&v.counters[Lists::kQueued]), unsigned(Lists::queue_cap(v)));
    const unsigned int warps = gridDim.x * kFuseWarps, me = blockIdx.x * kFuseWarps + warp;
    const unsigned int split = v.tb->fuse_split ? unsigned(v.tb->fuse_split) : fuse_split(halves, warps);
    const unsigned int sh = split >> 1, items = halves << sh;   // split = 1 << sh
    const unsigned int run = items / (kStaticItems * warps);    // items per run; 0: in turn
    FuseCtx& c = ctx[warp];
    int cur_s = -1;
    unsigned int i = run ? me * run : me, end = run ? min(i + run, items) : items;
    const unsigned int stride = run ? 1u : warps;
    uint2 next = i < end ? __ldcg(queue + (i >> sh)) : make_uint2(0u, 0u);
    while (i < items) {
        for (; i < end; i += stride) {
            const uint2 e = next;
            if (i + stride < end) next = __ldcg(queue + ((i + stride) >> sh));
            if (int(e.x) != cur_s) {
                cur_s = int(e.x);
                __syncwarp();
                load_ctx(Lists::ctx(v) + cur_s, c, lane);
                __syncwarp();
            }
            fuse_part<kFmt>(c, e.y, i & (split - 1u), split, lane);
        }
        if (!run) break;
        if (lane == 0) i = warps * run + atomicAdd(taken, run);
        i = __shfl_sync(0xffffffffu, i, 0);
        end = min(i + run, items);
        if (i < end) next = __ldcg(queue + (i >> sh));
    }
}

template <bool kVis>
static cudaError_t launch_fuse_of(const EngineView& v, int grid, int fmt, cudaStream_t st) {
    fuse_cull_kernel<kVis><<<grid, 256, 0, st>>>(v);   // grid-stride over all units of all sessions
    if (fmt == KF_TSDF_F32F32) fuse_kernel<kVis, KF_TSDF_F32F32><<<grid, 256, 0, st>>>(v);
    else if (fmt == KF_TSDF_F16U16) fuse_kernel<kVis, KF_TSDF_F16U16><<<grid, 256, 0, st>>>(v);
    else fuse_kernel<kVis, kAnyFormat><<<grid, 256, 0, st>>>(v);
    return cudaGetLastError();
}

cudaError_t launch_fuse(const EngineView& v, int grid, int fmt, cudaStream_t st) {
    return launch_fuse_of<false>(v, grid, fmt, st);
}

cudaError_t launch_fuse_vis(const EngineView& v, int grid, int fmt, cudaStream_t st) {
    return launch_fuse_of<true>(v, grid, fmt, st);
}

// ---- brick bounds ----
//
// bmin: lower bound of each 8^3 brick's distances (fusion's atomic minima).
// bdil: bmin widened to bricks {b, b+1}^3 (clamped), every brick a trilinear sample whose base
//       voxel lies in brick b can touch; the raycaster's brick-level skip test reads it.
// sdil: the same for 32^3 super-bricks: the minimum of bmin over bricks [4s, 4s + 4] per axis.
//       The raycaster reads the two small arrays (sdil stays in L1) to skip samples.
// Fusion keeps bdil and sdil equal to these minima as it lowers bmin (lower_brick_bound); the
// kernels below compute them from scratch after a volume is loaded.

// bdil[b] = min of bmin over bricks {b, b+1}^3 (clamped); nb^3 < 2^31, so 32-bit indices
__device__ __forceinline__ void dilate_brick(const int* __restrict__ m, int* bdil, int nb, int b) {
    const int bx = b % nb, byz = b / nb, by = byz % nb, bz = byz / nb;
    const int dx = bx + 1 < nb ? 1 : 0, dy = by + 1 < nb ? nb : 0, dz = bz + 1 < nb ? nb * nb : 0;
    const int* p = m + b;
    int k = min(min(__ldg(p), __ldg(p + dx)), min(__ldg(p + dy), __ldg(p + dy + dx)));
    k = min(k, min(min(__ldg(p + dz), __ldg(p + dz + dx)), min(__ldg(p + dz + dy), __ldg(p + dz + dy + dx))));
    bdil[b] = k;
}

// sdil of super-brick (sx, sy, sz): min of bmin over bricks [4s, 4s + 4] per axis (clamped),
// one warp
__device__ __forceinline__ int superbrick_bound(const int* bmin, int nb, int sx, int sy, int sz, int lane) {
    const int x0 = 4 * sx, y0 = 4 * sy, z0 = 4 * sz;
    int k = 0x7fffffff;
    for (int q = lane; q < 125; q += 32) {
        const int x = min(x0 + q % 5, nb - 1), y = min(y0 + (q / 5) % 5, nb - 1), z = min(z0 + q / 25, nb - 1);
        k = min(k, __ldg(bmin + (size_t(z) * nb + y) * nb + x));
    }
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) k = min(k, __shfl_xor_sync(0xffffffffu, k, off));
    return k;
}

__global__ void fill_key_kernel(int* a, long long count, int key) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < count; i += (long long)gridDim.x * blockDim.x)
        a[i] = key;
}

cudaError_t launch_init_bricks(int* bmin, int* bdil, int* sdil, int n, cudaStream_t st) {
    const int nb = n / 8, ns = (nb + 3) / 4;
    const long long nbricks = (long long)nb * nb * nb, nsuper = (long long)ns * ns * ns;
    const int k2 = 0x40000000;   // key of 2.0f (bits of a positive float)
    fill_key_kernel<<<148 * 4, 256, 0, st>>>(bmin, nbricks, k2);
    fill_key_kernel<<<148 * 4, 256, 0, st>>>(bdil, nbricks, k2);
    fill_key_kernel<<<148, 256, 0, st>>>(sdil, nsuper, k2);
    return cudaGetLastError();
}

// exact minimum over each brick's own 8^3 voxels (after a volume load), one warp per brick
template <class TF>
__global__ void rebuild_bricks_kernel(const TF* f, int n, int* bmin) {
    const int nb = n / 8;
    const long long total = (long long)nb * nb * nb;
    const int lane = threadIdx.x & 31;
    const long long warp = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long b = warp; b < total; b += nwarps) {
        const int bx = int(b % nb), by = int((b / nb) % nb), bz = int(b / ((long long)nb * nb));
        float m = 3.0e38f;
        for (int q = lane; q < 512; q += 32) {
            const int x = bx * 8 + (q & 7), y = by * 8 + ((q >> 3) & 7), z = bz * 8 + (q >> 6);
            m = fminf(m, load_f(f, (size_t(z) * n + y) * n + x));
        }
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) m = fminf(m, __shfl_xor_sync(0xffffffffu, m, off));
        if (lane == 0) bmin[b] = fkey(m);
    }
}

// bdil by the first blocks (one thread per brick), sdil by the rest (one warp per super-brick)
__global__ void __launch_bounds__(256) widen_kernel(const int* bmin, int* bdil, int* sdil, int nb, int dilate_blocks) {
    const int total = nb * nb * nb;
    if (int(blockIdx.x) < dilate_blocks) {
        for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < total; b += dilate_blocks * blockDim.x)
            dilate_brick(bmin, bdil, nb, b);
        return;
    }
    const int ns = (nb + 3) / 4, lane = threadIdx.x & 31;
    const int warp = ((blockIdx.x - dilate_blocks) * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = ((gridDim.x - dilate_blocks) * blockDim.x) >> 5;
    for (int b = warp; b < ns * ns * ns; b += nwarps) {
        const int k = superbrick_bound(bmin, nb, b % ns, (b / ns) % ns, b / (ns * ns), lane);
        if (lane == 0) sdil[b] = k;
    }
}

cudaError_t launch_widen_bricks(const int* bmin, int* bdil, int* sdil, int n, cudaStream_t st) {
    const int nb = n / 8;
    widen_kernel<<<148 * 8, 256, 0, st>>>(bmin, bdil, sdil, nb, 148 * 4);
    return cudaGetLastError();
}

cudaError_t launch_rebuild_bricks(const void* f, int fmt, int n, int* bmin, int* bdil, int* sdil, cudaStream_t st) {
    if (fmt == KF_TSDF_F16U16)
        rebuild_bricks_kernel<<<148 * 8, 256, 0, st>>>(static_cast<const __half*>(f), n, bmin);
    else
        rebuild_bricks_kernel<<<148 * 8, 256, 0, st>>>(static_cast<const float*>(f), n, bmin);
    return launch_widen_bricks(bmin, bdil, sdil, n, st);
}

// ---- stage fusion on a caller volume (kernel::fuse) ----
//
// The same cull, queue and fuse as a session's step, on scratch that the call brings.  The set-up
// launch writes what a session keeps: the voxel axes and the depth map's 16 x 16 tile maxima.  Bound
// by the queue's row updates, as a session's fusion.  One launch whose warps each tested and fused
// 32 consecutive blocks, without the maxima, was bound by the few warps that held the frustum's
// blocks: 808 us in the kernel at 640 x 480 into 512^3 f32, and up to 1 ms more per call in
// cudaMalloc and cudaFree; the call now takes 75 us, 41 of them kernels.

// the scratch of one call, carved from one allocation
struct StageFuseScratch {
    unsigned int* counters;   // [0] half units queued
    float* xs;
    float* zs;
    float* dmax;
    unsigned int* queue;      // pack_brick of each half unit that can update
};

static size_t stage_fuse_layout(int n, int w, int h, char* base, StageFuseScratch* s) {
    size_t at = 0;
    auto take = [&](size_t bytes) { const size_t o = at; at += (bytes + 255) & ~size_t(255); return base + o; };
    StageFuseScratch r;
    r.counters = reinterpret_cast<unsigned int*>(take(2 * sizeof(unsigned int)));
    r.xs = reinterpret_cast<float*>(take(sizeof(float) * n));
    r.zs = reinterpret_cast<float*>(take(sizeof(float) * n));
    r.dmax = reinterpret_cast<float*>(take(sizeof(float) * size_t((w + 15) / 16) * ((h + 15) / 16)));
    r.queue = reinterpret_cast<unsigned int*>(take(sizeof(unsigned int) * 2 * fuse_units(n)));
    if (s) *s = r;
    return at;
}

size_t stage_fuse_scratch(int n, int w, int h) { return stage_fuse_layout(n, w, h, nullptr, nullptr); }

// Block 0: counters and voxel axes (voxel_axes on the host: every product and sum rounded on its
// own, z accumulated step by step).  The other blocks: one warp per 16 x 16 tile of the depth map,
// its largest valid depth.
__global__ void __launch_bounds__(256) fuse_stage_setup_kernel(const float* depth, int w, int h, int n, float base,
                                                               float res, StageFuseScratch s) {
    const int tid = threadIdx.x;
    if (blockIdx.x == 0) {
        if (tid == 0) s.counters[0] = 0u;
        for (int i = tid; i < n; i += blockDim.x) s.xs[i] = __fadd_rn(base, __fmul_rn(float(i), res));
        if (tid == 0) {
            float z = __fsub_rn(base, res);
            for (int k = 0; k < n; ++k) {
                z = __fadd_rn(z, res);
                s.zs[k] = z;
            }
        }
        return;
    }
    const int lane = tid & 31, t16w = (w + 15) / 16, tiles = t16w * ((h + 15) / 16);
    const int t = (blockIdx.x - 1) * 8 + (tid >> 5);
    if (t >= tiles) return;
    const int x = (t % t16w) * 16 + (lane & 15), y0 = (t / t16w) * 16 + (lane >> 4);
    float m = 0.0f;
#pragma unroll
    for (int k = 0; k < 16; k += 2) {
        const float d = x < w && y0 + k < h ? __ldg(depth + size_t(y0 + k) * w + x) : 0.0f;
        if (depth_valid(d)) m = fmaxf(m, d);
    }
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
    if (lane == 0) s.dmax[t] = m;
}

// one thread per 32 x 8 x 8 unit, then one per half of the units that passed, as fuse_cull_kernel
__global__ void __launch_bounds__(256) fuse_stage_cull_kernel(const __grid_constant__ FuseCtx c, StageFuseScratch s) {
    __shared__ unsigned short list[256 * 4];
    __shared__ int packed;
    const int u0 = blockIdx.x * blockDim.x, tid = threadIdx.x, lane = tid & 31;
    int x0, j0, k0;
    unsigned int m = 0;
    if (u0 + tid < fuse_units(c.n)) {
        unit_origin(c.n, u0 + tid, x0, j0, k0);
        if (!block_culled(c, x0, 32, j0, k0)) m = unit_halves(c.n, x0);
    }
    const int count = block_pack(m, list, &packed);
    for (int i = tid & ~31; i < count; i += 256) {
        const int code = i + lane < count ? list[i + lane] : 0, u = u0 + (code >> 2);
        unit_origin(c.n, u, x0, j0, k0);
        const bool keep = i + lane < count && !block_culled(c, x0 + 16 * (code & 3), 16, j0, k0);
        const unsigned int km = __ballot_sync(0xffffffffu, keep);
        if (km == 0) continue;
        unsigned int slot = 0;
        if (lane == 0) slot = atomicAdd(s.counters, unsigned(__popc(km)));
        slot = __shfl_sync(0xffffffffu, slot, 0);
        if (keep) s.queue[slot + __popc(km & ((1u << lane) - 1u))] = pack_brick((x0 >> 3) + 2 * (code & 3), j0 >> 3, k0 >> 3);
    }
}

template <int kFmt>
__global__ void __launch_bounds__(256, 4) fuse_stage_kernel(const __grid_constant__ FuseCtx c, StageFuseScratch s) {
    const int lane = threadIdx.x & 31;
    const unsigned int halves = __ldcg(s.counters), warps = gridDim.x * kFuseWarps;
    const unsigned int split = fuse_split(halves, warps), sh = split >> 1, items = halves << sh;
    unsigned int i = blockIdx.x * kFuseWarps + (threadIdx.x >> 5);
    unsigned int next = i < items ? __ldcg(s.queue + (i >> sh)) : 0u;
    for (; i < items; i += warps) {
        const unsigned int e = next;
        if (i + warps < items) next = __ldcg(s.queue + ((i + warps) >> sh));
        fuse_part<kFmt>(c, e, i & (split - 1u), split, lane);
    }
}

cudaError_t stage_fuse(const float* depth, int w, int h, const float* k, const kf_volume* vol, const float* pose,
                       float min_d, float max_d, void* scratch, cudaStream_t st) {
    StageFuseScratch s;
    stage_fuse_layout(vol->n, w, h, static_cast<char*>(scratch), &s);
    FuseCtx c{};
    c.depth = depth;
    c.dmax = s.dmax;
    c.t16w = (w + 15) / 16;
    c.w = w;
    c.h = h;
    c.fx = k[0]; c.fy = k[4]; c.cx = k[6]; c.cy = k[7];
    c.min_d = min_d; c.max_d = max_d; c.mu = vol->mu; c.max_w = vol->max_weight;
    c.n = vol->n;
    c.nb = vol->n / 8;
    c.fmt = vol->format;
    c.F = vol->f;
    c.W = vol->w;
    c.xs = s.xs;
    c.zs = s.zs;
    c.bmin = nullptr;
    // inverse of the rigid pose: R^T, -R^T t
    for (int col = 0; col < 3; ++col)
        for (int row = 0; row < 3; ++row) c.iR[col * 3 + row] = pose[row * 4 + col];
    for (int row = 0; row < 3; ++row)
        c.it[row] = -(c.iR[row] * pose[12] + c.iR[3 + row] * pose[13] + c.iR[6 + row] * pose[14]);
    const float res = vol->width / float(vol->n - 1), base = -vol->width * 0.5f;
    const int tiles = c.t16w * ((h + 15) / 16);
    fuse_stage_setup_kernel<<<1 + (tiles + 7) / 8, 256, 0, st>>>(depth, w, h, vol->n, base, res, s);
    fuse_stage_cull_kernel<<<(fuse_units(vol->n) + 255) / 256, 256, 0, st>>>(c, s);
    if (vol->format == KF_TSDF_F16U16) fuse_stage_kernel<KF_TSDF_F16U16><<<148 * 4, 256, 0, st>>>(c, s);
    else fuse_stage_kernel<KF_TSDF_F32F32><<<148 * 4, 256, 0, st>>>(c, s);
    return cudaGetLastError();
}

// ---- initialisation {f = 2, w = 0} (project/src/voxel_grid.h:8-15) and layout conversion ----

__global__ void init_f32_kernel(float4* f, float4* w, long long nvec) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nvec; i += (long long)gridDim.x * blockDim.x) {
        f[i] = make_float4(2.f, 2.f, 2.f, 2.f);
        w[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
}
__global__ void init_f16_kernel(uint4* f, uint4* w, long long nvec) {
    const __half two = __float2half_rn(2.0f);
    const unsigned short tb = *reinterpret_cast<const unsigned short*>(&two);
    const unsigned int pair = (unsigned int)tb | ((unsigned int)tb << 16);
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nvec; i += (long long)gridDim.x * blockDim.x) {
        f[i] = make_uint4(pair, pair, pair, pair);
        w[i] = make_uint4(0u, 0u, 0u, 0u);
    }
}
__global__ void init_tail_kernel(void* f, void* w, long long start, long long nvox, int fmt) {
    for (long long i = start + blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nvox; i += (long long)gridDim.x * blockDim.x) {
        if (fmt == KF_TSDF_F16U16) {
            static_cast<__half*>(f)[i] = __float2half_rn(2.0f);
            static_cast<uint16_t*>(w)[i] = 0;
        } else {
            static_cast<float*>(f)[i] = 2.0f;
            static_cast<float*>(w)[i] = 0.0f;
        }
    }
}

cudaError_t launch_init_volume(void* f, void* w, long long nvox, int fmt, cudaStream_t st) {
    const int per = fmt == KF_TSDF_F16U16 ? 8 : 4;
    const long long nvec = nvox / per;
    const int grid = 148 * 8;
    if (nvec > 0) {
        if (fmt == KF_TSDF_F16U16)
            init_f16_kernel<<<grid, 256, 0, st>>>(static_cast<uint4*>(f), static_cast<uint4*>(w), nvec);
        else
            init_f32_kernel<<<grid, 256, 0, st>>>(static_cast<float4*>(f), static_cast<float4*>(w), nvec);
    }
    if (nvec * per < nvox) init_tail_kernel<<<1, 256, 0, st>>>(f, w, nvec * per, nvox, fmt);
    return cudaGetLastError();
}

__global__ void export_kernel(const void* f, const void* w, long long nvox, int fmt, float2* dst) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nvox; i += (long long)gridDim.x * blockDim.x) {
        float a, b;
        if (fmt == KF_TSDF_F16U16) {
            a = __half2float(static_cast<const __half*>(f)[i]);
            b = float(static_cast<const uint16_t*>(w)[i]) * (1.0f / KF_WEIGHT_SCALE);
        } else {
            a = static_cast<const float*>(f)[i];
            b = static_cast<const float*>(w)[i];
        }
        dst[i] = make_float2(a, b);
    }
}

__global__ void import_kernel(const float2* src, void* f, void* w, long long nvox, int fmt) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nvox; i += (long long)gridDim.x * blockDim.x) {
        const float2 v = src[i];
        if (fmt == KF_TSDF_F16U16) {
            static_cast<__half*>(f)[i] = __float2half_rn(v.x);
            static_cast<uint16_t*>(w)[i] = uint16_t(fminf(fmaxf(rintf(v.y * KF_WEIGHT_SCALE), 0.0f), 65535.0f));
        } else {
            static_cast<float*>(f)[i] = v.x;
            static_cast<float*>(w)[i] = v.y;
        }
    }
}

cudaError_t launch_export_interleaved(const void* f, const void* w, long long nvox, int fmt, float* dst, cudaStream_t st) {
    export_kernel<<<148 * 8, 256, 0, st>>>(f, w, nvox, fmt, reinterpret_cast<float2*>(dst));
    return cudaGetLastError();
}
cudaError_t launch_import_interleaved(const float* src, void* f, void* w, long long nvox, int fmt, cudaStream_t st) {
    import_kernel<<<148 * 8, 256, 0, st>>>(reinterpret_cast<const float2*>(src), f, w, nvox, fmt);
    return cudaGetLastError();
}

}  // namespace kf
