// Frame-to-model tracking: projective ICP + photometric normal equations
// (Tracking/Reduction.cu: ICPReduce 212-375, RGBReduction 377-627) and the
// coarse-to-fine Gauss-Newton loop of Tracker::ComputeSE3
// (Tracking/Tracking.cc:296-409), kept entirely on the device.
//
// One iteration has two passes:
//   pass A: per pixel, the ICP row (point-to-plane, 7 wide) and the RGB
//           correspondence search; ICP products and the RGB count / sum of
//           squared differences are reduced.  The RGB correspondences go to
//           lists, one per warp, in the order the warp met them.  The current
//           frame's per-pixel inputs are staged in shared memory by bulk
//           copies in 256-pixel chunks.
//   pass B: per correspondence, the photometric row weighted by the robust
//           scale sigma from pass A; products reduced.  Then A x = b is
//           solved in FP64 (LDL^T) and the SE(3) exponential applied, with
//           the reference's failure and acceptance tests.
// Reductions are deterministic: fixed per-thread pixel sets, warp shuffles,
// block sums in shared memory, block sums added per group of kTrackCluster
// blocks and the groups in order in FP64 (no atomics on values).
//
// A session alone runs all iterations of a frame in one cooperative kernel
// (k_track_loop).  Sessions sharing the GPU run a kernel per pass, on a
// quarter of the blocks and with half the registers, so that several
// sessions' passes run side by side (k_track_a_grp / k_track_b_grp).  Both
// walk the same logical grid and add in the same order, and this file is
// compiled without contraction of multiplies and adds into FMAs, so both
// compute the same bits.
#include <cooperative_groups.h>

#include <algorithm>
#include <mutex>

#include "fb_async.cuh"
#include "fb_fused.cuh"
#include "fb_internal.h"

namespace cg = cooperative_groups;

namespace fb {

// ------------------------------------------------------------ row builders
//
// The reference evaluates a few float expressions in double (Reduction.cu:
// (float)(1.0 / (double)z), (int)((double)f + 0.5), (float)((double)f + 0.5),
// (double)dx / 9.0, (double)x < c).  Their float equivalents below give the
// same bits for every float input:
//   - a quotient or sum of floats computed in double and rounded to float is
//     the IEEE float quotient or sum (double rounding is innocuous when the
//     wide format has at least 2p + 2 bits: 53 >= 50; f + 0.5 is exact in
//     double where it matters), hence __frcp_rn, __fdiv_rn, __fadd_rn;
//   - (int)((double)f + 0.5) truncates f + 0.5; the float sum rounded toward
//     zero lies between that integer and the exact sum, so it truncates to
//     the same integer (saturation and NaN -> 0 as the double conversion);
//   - (double)x < c for a double c that is not a float holds exactly when x
//     is below the smallest float above c (1e-3; the 0.1 of the photometric
//     distance, whose float is that smallest one).
__device__ __forceinline__ int trunc_half_up(float f) { return __float2int_rz(__fadd_rz(f, 0.5f)); }
constexpr float kBelow1em3 = 0.001f;   // (double)x < 1e-3  <=>  x < 0.001f
// Square roots compared with a constant: the correctly rounded root is
// monotone, so fsq(x) <= 0.1f, fsq(x) < 0.1f and fsq(x) < 0.6f hold exactly
// up to one largest x each (NaN fails both forms).
__device__ __forceinline__ bool sqrt_le_0p1(float x) { return x <= __int_as_float(0x3c23d70b); }
__device__ __forceinline__ bool sqrt_lt_0p1(float x) { return x <= __int_as_float(0x3c23d709); }
__device__ __forceinline__ bool sqrt_lt_0p6(float x) { return x <= __int_as_float(0x3eb851eb); }
// A Sobel value / 9: one reciprocal and Markstein's correction (fd_rcp).
__device__ __forceinline__ float ninth(int d) { return fd_rcp((float)d, 9.0f, __int_as_float(0x3de38e39)); }
__device__ __forceinline__ float below_1em6() { return __int_as_float(0x358637be); }   // (double)x < 1e-6

// Photometric correspondences are packed in 32 bits: last-frame pixel
// (u, v) and the gray difference d (-254..255, as d + 255 in 1..510):
// v << 21 | u << 9 | (d + 255).  Images are at most 4096 x 2048; the low 9
// bits are never all ones, so -1 (all ones) marks "no correspondence".
// A correspondence list entry is {the pixel's Sobel derivatives (uint16) dx | dy << 16, pack_corr}.
__device__ __forceinline__ int pack_corr(int u, int v, int d255) {
    return (int)(((unsigned)v << 21) | ((unsigned)u << 9) | (unsigned)d255);
}
__device__ __forceinline__ int corr_u(int c) { return (int)(((unsigned)c >> 9) & 4095u); }
__device__ __forceinline__ int corr_v(int c) { return (int)((unsigned)c >> 21); }

// ICPReduce::searchPoint + getRow (Reduction.cu:227-286).  Returns false when
// the pixel has no correspondence.  Decisions use the order-exact float ops.
__device__ __forceinline__ bool icp_row(const TrackLevel& L, const DevPose& cur, const DevPose& last, int x,
                                        int y, float row[7]) {
    const size_t i = (size_t)y * L.vp + x;
    float4 vc4 = L.vcurr[i];
    f3 vcurr_c = xyz(vc4);
    if (isnan(vcurr_c.x) || vcurr_c.z < kBelow1em3) return false;
    f3 vcurr_g = add3(mv(cur.R, vcurr_c), cur.t);
    f3 vcurr_p = mv(last.Rinv, sub3(vcurr_g, last.t));
    float invz = __frcp_rn(vcurr_p.z);
    int u = trunc_half_up(fa(fm(fm(vcurr_p.x, invz), L.k.fx), L.k.cx));
    int v = trunc_half_up(fa(fm(fm(vcurr_p.y, invz), L.k.fy), L.k.cy));
    if (u < 0 || v < 0 || u >= L.W || v >= L.H) return false;
    const size_t j = (size_t)v * L.vp + u;
    f3 vlast_c = xyz(L.vlast[j]);
    f3 vlast_g = add3(mv(last.R, vlast_c), last.t);
    f3 ncurr_c = xyz(L.ncurr[i]);
    f3 ncurr_g = mv(cur.R, ncurr_c);
    f3 nlast_c = xyz(L.nlast[j]);
    f3 nlast_g = mv(last.R, nlast_c);
    const f3 gap = sub3(vlast_g, vcurr_g), turn = cross3(ncurr_g, nlast_g);
    if (!(sqrt_lt_0p6(dot3(turn, turn)) && sqrt_le_0p1(dot3(gap, gap)) && !isnan(ncurr_c.x) && !isnan(nlast_c.x)))
        return false;
    f3 nl = mv(last.Rinv, nlast_g);
    f3 vcl = mv(last.Rinv, sub3(vcurr_g, last.t));
    f3 vll = mv(last.Rinv, sub3(vlast_g, last.t));
    f3 c = cross3(nl, vll);
    row[0] = -nl.x;
    row[1] = -nl.y;
    row[2] = -nl.z;
    row[3] = c.x;
    row[4] = c.y;
    row[5] = c.z;
    row[6] = dot3(neg3(nl), sub3(vcl, vll));
    return true;
}

// RGBReduction::FindCorresp (Reduction.cu:404-451).  Returns the packed
// correspondence (pack_corr) of last-frame pixel (u, v), or -1.
__device__ __forceinline__ int rgb_corresp(const TrackLevel& L, const DevPose& cur, const DevPose& last, int x,
                                           int y) {
    const int W = L.W, H = L.H;
    if (L.rgbok) {
        // border, window and gradient tests precomputed per frame
        if (!L.rgbok[(size_t)y * L.sp + x]) return -1;
    } else {
        if (!(x >= 5 && x < W - 5 && y >= 5 && y < H - 5)) return -1;
        // the window is y-2..y+1, x-2..x+1 (Reduction.cu:416-417), loaded together
        bool any0 = false;
#pragma unroll
        for (int q = 0; q < 16; ++q) any0 |= L.gcurr[(size_t)(y - 2 + q / 4) * L.gp + x - 2 + q % 4] == 0;
        if (any0) return -1;
        int gx = L.dx[(size_t)y * L.sp + x], gy = L.dy[(size_t)y * L.sp + x];
        if (gx == 0 && gy == 0) return -1;  // sqrtf(gx*gx + gy*gy) > 0
    }
    float4 vcurr = L.vcurr[(size_t)y * L.vp + x];
    if (isnan(vcurr.x)) return -1;
    f3 vcurr_g = add3(mv(cur.R, xyz(vcurr)), cur.t);
    f3 vcl = mv(last.Rinv, sub3(vcurr_g, last.t));
    float pu = fa(fd(fm(L.k.fx, vcl.x), vcl.z), L.k.cx);
    float pv = fa(fd(fm(L.k.fy, vcl.y), vcl.z), L.k.cy);
    int u = __float2int_rd(__fadd_rn(pu, 0.5f));
    int v = __float2int_rd(__fadd_rn(pv, 0.5f));
    if (!(u >= 0 && v >= 0 && u < W && v < H)) return -1;
    float4 vlast = L.vlast[(size_t)v * L.vp + u];
    if (isnan(vlast.x)) return -1;
    float ddx = fs(vlast.x, vcurr.x), ddy = fs(vlast.y, vcurr.y), ddz = fs(vlast.z, vcurr.z),
          ddw = fs(vlast.w, vcurr.w);
    if (!sqrt_lt_0p1(fa(fa(fa(fm(ddx, ddx), fm(ddy, ddy)), fm(ddz, ddz)), fm(ddw, ddw)))) return -1;
    int gl = L.glast[(size_t)v * L.gp + u];
    if (gl == 0) return -1;
    int diff = (int)L.gcurr[(size_t)y * L.gp + x] - gl;
    return pack_corr(u, v, diff + 255);
}

// The memory inputs of one photometric row: the last frame's vertex at the
// correspondence, the current pixel's derivatives and the packed value.
struct RgbIn {
    float4 vlast;
    int dx, dy, packed;
};

__device__ __forceinline__ RgbIn rgb_fetch(const TrackLevel& L, int x, int y, int packed) {
    RgbIn in;
    in.vlast = L.vlast[corr_v(packed) * L.vp + corr_u(packed)];
    const int k = y * L.sp + x;
    in.dx = L.dx[k];
    in.dy = L.dy[k];
    in.packed = packed;
    return in;
}

// The fetch of correspondence list entry e (the pixel's derivatives
// (uint16) dx | dy << 16, packed value): only the last vertex at the
// correspondence is gathered.
__device__ __forceinline__ RgbIn rgb_fetch_entry(const TrackLevel& L, int2 e) {
    RgbIn in;
    in.vlast = L.vlast[corr_v(e.y) * L.vp + corr_u(e.y)];
    in.dx = (int)(int16_t)(e.x & 0xffff);
    in.dy = e.x >> 16;
    in.packed = e.y;
    return in;
}

// RGBReduction::GetRow (Reduction.cu:471-508) from fetched inputs, in two
// parts: the row's six direction values, which need no weight, and the weight
// by the robust scale.
struct RgbDir {
    f3 left, c;
};

__device__ __forceinline__ RgbDir rgb_dir(f3 vlast, int dx, int dy, const TrackLevel& L, const DevPose& cur,
                                          const DevPose& last) {
    f3 point = mv(cur.Rinv, sub3(add3(mv(last.R, vlast), last.t), cur.t));
    float gx = ninth(dx);
    float gy = ninth(dy);
    float invz = __frcp_rn(point.z);
    RgbDir d;
    d.left.x = gx * L.k.fx * invz;
    d.left.y = gy * L.k.fy * invz;
    d.left.z = -(d.left.x * point.x + d.left.y * point.y) * invz;
    d.c = cross3(point, d.left);
    return d;
}

__device__ __forceinline__ void rgb_weighted(const RgbDir& d, int diff, float sigma, float row[7]) {
    float w = sigma + (float)abs(diff);
    w = w < kBelow1em3 ? 1.0f : __frcp_rn(w);
    if (sigma < below_1em6()) w = 1.0f;
    row[0] = w * d.left.x;
    row[1] = w * d.left.y;
    row[2] = w * d.left.z;
    row[3] = w * d.c.x;
    row[4] = w * d.c.y;
    row[5] = w * d.c.z;
    row[6] = -w * (float)diff;
}

__device__ __forceinline__ void rgb_row_of(const RgbIn& in, const TrackLevel& L, const DevPose& cur,
                                           const DevPose& last, float sigma, float row[7]) {
    rgb_weighted(rgb_dir(xyz(in.vlast), in.dx, in.dy, L, cur, last), (in.packed & 511) - 255, sigma, row);
}

// RGBReduction::GetRow of the correspondence `packed` of pixel (x, y).
__device__ __forceinline__ void rgb_row(const TrackLevel& L, const DevPose& cur, const DevPose& last, int x, int y,
                                        int packed, float sigma, float row[7]) {
    rgb_row_of(rgb_fetch(L, x, y, packed), L, cur, last, sigma, row);
}

// Pose-independent inputs of one pixel for pass A (staged in shared memory
// by PixelStage).
struct PixelIn {
    float4 vc;      // current vertex
    float3 nc;      // current normal (xyz)
    int ok;         // photometric eligibility (border, window, gradient)
    int gc;         // current gray value
    int dxy;        // Sobel derivatives: (uint16) dx | dy << 16
};

// Pass A's current-frame inputs staged in shared memory by bulk copies
// (cp.async.bulk, this GPU's own memory, no multicast).  A chunk is one
// logical block's 256 consecutive pixels of one pass over the image (the
// frame buffers have pitch == width, so a chunk is one contiguous range of
// each map): vertices and normals (4 KB each), the Sobel derivatives
// (512 B each), photometric eligibility and gray (256 B each; the derivative
// and byte rows are rounded up to 16 B at the image's end, inside the
// allocations, which are 256-byte multiples).  Two buffers: chunk c + 2 is
// copied while chunk c + 1 is processed.
struct PixelStage {
    float4 v[2][256];
    float4 n[2][256];
    int16_t dx[2][256];
    int16_t dy[2][256];
    uint8_t ok[2][256];
    uint8_t g[2][256];
    uint64_t bar[2];
};

// Thread 0: copy the chunk of pixels [start, min(start + 256, N)) into
// buffer `buf`, completing on its barrier.
__device__ __forceinline__ void stage_chunk(PixelStage& S, int buf, const TrackLevel& L, int start, int N) {
    const int cnt = min(256, N - start);
    const uint32_t b16 = (uint32_t)cnt * 16u, b1 = ((uint32_t)cnt + 15u) & ~15u;
    const uint32_t b2 = ((uint32_t)cnt * 2u + 15u) & ~15u;
    fence_proxy_async_smem();
    mbar_arrive_expect_tx(&S.bar[buf], 2u * b16 + 2u * b2 + 2u * b1);
    bulk_copy_g2s(S.v[buf], L.vcurr + start, b16, &S.bar[buf]);
    bulk_copy_g2s(S.n[buf], L.ncurr + start, b16, &S.bar[buf]);
    bulk_copy_g2s(S.dx[buf], L.dx + start, b2, &S.bar[buf]);
    bulk_copy_g2s(S.dy[buf], L.dy + start, b2, &S.bar[buf]);
    bulk_copy_g2s(S.ok[buf], L.rgbok + start, b1, &S.bar[buf]);
    bulk_copy_g2s(S.g[buf], L.gcurr + start, b1, &S.bar[buf]);
}

// Every thread: wait for buffer `buf`'s fill number `use` (bounded); then
// read pixel t of the chunk.  Returns false in every thread of the block
// when any thread's wait gave up.
__device__ __forceinline__ bool take_chunk(PixelStage& S, int buf, uint32_t use) {
    const bool ok = mbar_wait(&S.bar[buf], use & 1u);
    return !__syncthreads_or(!ok);
}

// The chunks of a group-form block in processing order: groups j of the
// block, the group's kTrackCluster logical blocks r, their passes k over the
// image while the chunk starts inside it.  start < 0: no chunk left.
struct ChunkCursor {
    int j, r, k, start;
    __device__ __forceinline__ int start_of(int bx, int gpc, int S) const {
        return ((bx * gpc + j) * kTrackCluster + r) * 256 + k * S;
    }
    // the first chunk at or after (j, r, k)
    __device__ __forceinline__ void settle(int bx, int gpc, int NG, int iters, int S, int N) {
        for (;;) {
            if (j >= gpc || bx * gpc + j >= NG) {
                start = -1;
                return;
            }
            if (k < iters) {
                start = start_of(bx, gpc, S);
                if (start < N) return;
            }
            k = 0;
            if (++r == kTrackCluster) {
                r = 0;
                ++j;
            }
            if (start_of(bx, gpc, S) >= N) {   // later logical blocks start later still
                start = -1;
                return;
            }
        }
    }
};

__device__ __forceinline__ PixelIn staged_pixel(const PixelStage& S, int buf, int t) {
    PixelIn in;
    in.vc = S.v[buf][t];
    const float4 n = S.n[buf][t];
    in.nc = make_float3(n.x, n.y, n.z);
    in.ok = S.ok[buf][t];
    in.gc = S.g[buf][t];
    in.dxy = (int)(uint16_t)S.dx[buf][t] | ((int)S.dy[buf][t] << 16);
    return in;
}

// icp_row and rgb_corresp of one pixel together (same arithmetic, same
// decisions), with the pose-independent loads done by the caller and the four
// pose-dependent gathers (last vertex and normal at the ICP projection, last
// vertex and gray value at the photometric projection) issued together.
// Needs L.rgbok.  Returns whether the ICP row is valid; *rgb = packed
// correspondence or -1, *vphoto = the last vertex at it.
__device__ __forceinline__ bool pixel_pass_a(const TrackLevel& L, const DevPose& cur, const DevPose& last,
                                             const PixelIn& in, float row[7], int* rgb, f3* vphoto = nullptr) {
    const f3 vcurr_c = xyz(in.vc);
    const bool vnan = isnan(vcurr_c.x);
    const f3 vcurr_g = add3(mv(cur.R, vcurr_c), cur.t);
    // ICP projection (ICPReduce::searchPoint, Reduction.cu:227-250)
    int ju = -1;
    if (!vnan && !(vcurr_c.z < kBelow1em3)) {
        const f3 vcurr_p = mv(last.Rinv, sub3(vcurr_g, last.t));
        const float invz = __frcp_rn(vcurr_p.z);
        const int u = trunc_half_up(fa(fm(fm(vcurr_p.x, invz), L.k.fx), L.k.cx));
        const int v = trunc_half_up(fa(fm(fm(vcurr_p.y, invz), L.k.fy), L.k.cy));
        if (!(u < 0 || v < 0 || u >= L.W || v >= L.H)) ju = v * L.vp + u;
    }
    // photometric projection (RGBReduction::FindCorresp, Reduction.cu:404-451)
    int jr = -1, ur = 0, vr = 0;
    if (in.ok && !vnan) {
        const f3 vcl = mv(last.Rinv, sub3(vcurr_g, last.t));
        const float pu = fa(fd(fm(L.k.fx, vcl.x), vcl.z), L.k.cx);
        const float pv = fa(fd(fm(L.k.fy, vcl.y), vcl.z), L.k.cy);
        ur = __float2int_rd(__fadd_rn(pu, 0.5f));
        vr = __float2int_rd(__fadd_rn(pv, 0.5f));
        if (ur >= 0 && vr >= 0 && ur < L.W && vr < L.H) jr = vr * L.vp + ur;
    }
    const float nanf_ = qnan();
    const float4 vl4 = ju >= 0 ? L.vlast[ju] : make_float4(nanf_, nanf_, nanf_, nanf_);
    const float4 nl4 = ju >= 0 ? L.nlast[ju] : make_float4(nanf_, nanf_, nanf_, nanf_);
    // the two projections mostly meet the same pixel: one gather then
    float4 vr4 = jr >= 0 && jr != ju ? L.vlast[jr] : make_float4(nanf_, nanf_, nanf_, nanf_);
    const int gl = jr >= 0 ? (int)L.glast[vr * L.gp + ur] : 0;
    if (jr >= 0 && jr == ju) vr4 = vl4;
    if (vphoto) *vphoto = xyz(vr4);
    // photometric residual
    *rgb = -1;
    if (jr >= 0 && !isnan(vr4.x)) {
        const float ddx = fs(vr4.x, in.vc.x), ddy = fs(vr4.y, in.vc.y), ddz = fs(vr4.z, in.vc.z),
                    ddw = fs(vr4.w, in.vc.w);
        if (sqrt_lt_0p1(fa(fa(fa(fm(ddx, ddx), fm(ddy, ddy)), fm(ddz, ddz)), fm(ddw, ddw))) && gl != 0) *rgb = pack_corr(ur, vr, in.gc - gl + 255);
    }
    // ICP row (ICPReduce::getRow, Reduction.cu:252-286)
    if (ju < 0) return false;
    const f3 vlast_c = xyz(vl4);
    const f3 vlast_g = add3(mv(last.R, vlast_c), last.t);
    const f3 ncurr_c = mk3(in.nc.x, in.nc.y, in.nc.z);
    const f3 ncurr_g = mv(cur.R, ncurr_c);
    const f3 nlast_c = xyz(nl4);
    const f3 nlast_g = mv(last.R, nlast_c);
    const f3 gap = sub3(vlast_g, vcurr_g), turn = cross3(ncurr_g, nlast_g);
    if (!(sqrt_lt_0p6(dot3(turn, turn)) && sqrt_le_0p1(dot3(gap, gap)) && !isnan(ncurr_c.x) && !isnan(nlast_c.x)))
        return false;
    const f3 nl = mv(last.Rinv, nlast_g);
    const f3 vcl = mv(last.Rinv, sub3(vcurr_g, last.t));
    const f3 vll = mv(last.Rinv, sub3(vlast_g, last.t));
    const f3 c = cross3(nl, vll);
    row[0] = -nl.x;
    row[1] = -nl.y;
    row[2] = -nl.z;
    row[3] = c.x;
    row[4] = c.y;
    row[5] = c.z;
    row[6] = dot3(neg3(nl), sub3(vcl, vll));
    return true;
}

__device__ __forceinline__ void add_products(const float row[7], float acc[29]) {
    int n = 0;
#pragma unroll
    for (int i = 0; i < 7; ++i)
#pragma unroll
        for (int j = i; j < 7; ++j) acc[n++] += row[i] * row[j];
    acc[28] += 1.0f;
}

// Pass B's rows of one warp segment (n entries): lane l adds the rows of
// entries l, l + 32, ... in that order.
__device__ __forceinline__ void add_segment_rows(const TrackLevel& L, const DevPose& cur, const DevPose& last,
                                                     float sigma, const int2* seg, int n, int lane, float acc[29]) {
    for (int i = lane; i < n; i += 32) {
        float row[7];
        rgb_row_of(rgb_fetch_entry(L, seg[i]), L, cur, last, sigma, row);
        add_products(row, acc);
    }
}

// ------------------------------------------------------------- reductions

// Warp sums of the 29 per-thread values of the normal equations by recursive
// halving: at every step a lane keeps one half of its values, sends the other
// half to its partner and adds what it receives (31 shuffles in all).  Lane l
// then holds the warp sum of value l, added as the halving tree over the lanes.
__device__ __forceinline__ float warp_sum29(const float (&v)[29]) {
    const int lane = threadIdx.x & 31;
    float a[32];
#pragma unroll
    for (int k = 0; k < 29; ++k) a[k] = v[k];
    a[29] = a[30] = a[31] = 0.f;
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) {
        const bool up = (lane & off) != 0;
#pragma unroll
        for (int k = 0; k < off; ++k) {
            const float send = up ? a[k] : a[k + off];
            const float keep = up ? a[k + off] : a[k];
            a[k] = keep + __shfl_xor_sync(0xffffffffu, send, off);
        }
    }
    return a[0];
}

// Block-wide sum of the 29 values: the warps' sums added in warp order by warp
// 0.  Result: value l in lane l (< 29) of warp 0.  Deterministic.
__device__ __forceinline__ float block_sum29(const float (&v)[29], float* smem /* [8][32] */) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    smem[wid * 32 + lane] = warp_sum29(v);
    __syncthreads();
    float r = 0.f;
    if (wid == 0)
        for (int w = 0; w < nw; ++w) r += smem[w * 32 + lane];
    return r;
}

// The same with the eight warps' sums added as a halving tree (the single-step
// entry points' order).
__device__ __forceinline__ float block_tree29(const float (&v)[29], float* smem /* [8][32] */) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    smem[wid * 32 + lane] = warp_sum29(v);
    __syncthreads();
    const float* w = smem + lane;
    return wid == 0 ? ((w[0] + w[128]) + (w[64] + w[192])) + ((w[32] + w[160]) + (w[96] + w[224])) : 0.f;
}

__device__ __forceinline__ long long block_sum_ll(long long v, long long* smem) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    __syncthreads();
    if (lane == 0) smem[wid] = v;
    __syncthreads();
    if (wid == 0) {
        v = lane < nw ? smem[lane] : 0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    }
    return v;
}

// Ticket increment with release (this block's prior writes, ordered before it
// by a block barrier) and acquire (the writes of the blocks that incremented
// before) semantics at GPU scope.
__device__ __forceinline__ unsigned int ticket_acq_rel(unsigned int* t) {
    unsigned int old;
    asm volatile("atom.add.acq_rel.gpu.u32 %0, [%1], 1;" : "=r"(old) : "l"(t) : "memory");
    return old;
}

// Last-block-done: returns true in every thread of the last block to finish.
__device__ __forceinline__ bool last_block(unsigned int* ticket) {
    __shared__ bool is_last;
    __syncthreads();
    if (threadIdx.x == 0) is_last = ticket_acq_rel(ticket) == gridDim.x - 1;
    __syncthreads();
    return is_last;
}

// ----------------------------------------------------------- FP64 solver

__device__ __forceinline__ void mat4_mul(const double* A, const double* B, double* C) {
    double T[16];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            double s = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) s += A[i * 4 + k] * B[k * 4 + j];
            T[i * 4 + j] = s;
        }
#pragma unroll
    for (int i = 0; i < 16; ++i) C[i] = T[i];
}

__device__ __forceinline__ void mat4_rigid_inv(const double* A, double* B) {
    double T[16];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) T[i * 4 + j] = A[j * 4 + i];
#pragma unroll
    for (int i = 0; i < 3; ++i)
        T[i * 4 + 3] = -(T[i * 4 + 0] * A[3] + T[i * 4 + 1] * A[7] + T[i * 4 + 2] * A[11]);
    T[12] = T[13] = T[14] = 0;
    T[15] = 1;
#pragma unroll
    for (int i = 0; i < 16; ++i) B[i] = T[i];
}

__device__ double euler_sin_norm(const double* T) {
    double a = atan2(-T[6], T[10]);
    double b = atan2(T[2], sqrt(T[0] * T[0] + T[1] * T[1]));
    double c = atan2(-T[1], T[0]);
    double sa = sin(a), sb = sin(b), sc = sin(c);
    return sqrt(sa * sa + sb * sb + sc * sc);
}

// ------------------------------------------------------------------ kernels

__device__ __forceinline__ void track_begin_body(const BlockCtx&, TrackState* st, TrackSync* sync, unsigned step) {
    track_begin(st, sync, step);
}
__global__ void k_track_begin(TrackState* st, TrackSync* sync, unsigned step) {
    if (threadIdx.x == 0) track_begin(st, sync, step);
}
FB_FUSED_KERNEL(k_track_begin, track_begin_body, 32)

// Fixed-order FP64 sum of nv values over nb block partials laid out as
// partials[b * stride + v], computed by the whole block: thread t sums value
// (t % 32) over the block chunk (t / 32), then the 8 chunk sums are added in
// order.  Deterministic for a given nb.  out: shared array of nv doubles.
__device__ void reduce_partials(const float* partials, int nb, int stride, int nv, double* out,
                                double* scratch /* [8][32] shared */) {
    const int v = threadIdx.x & 31, c = threadIdx.x >> 5, nc = blockDim.x >> 5;
    const int per = (nb + nc - 1) / nc;
    for (int v0 = 0; v0 < nv; v0 += 32) {
        double s = 0;
        if (v0 + v < nv) {
            const int b0 = c * per, b1 = min(nb, b0 + per);
            for (int b = b0; b < b1; b += 16) {   // loaded together, added in order
                float x[16];
#pragma unroll
                for (int q = 0; q < 16; ++q)
                    if (b + q < b1) x[q] = __ldcg(partials + (size_t)(b + q) * stride + v0 + v);
#pragma unroll
                for (int q = 0; q < 16; ++q)
                    if (b + q < b1) s += (double)x[q];
            }
        }
        scratch[c * 32 + v] = s;
        __syncthreads();
        if (c == 0 && v0 + v < nv) {
            double t = 0;
            for (int q = 0; q < nc; ++q) t += scratch[q * 32 + v];
            out[v0 + v] = t;
        }
        __syncthreads();
    }
}

// Bytes of the per-warp correspondence segments for n pixels: every warp of
// the pass-A grid gets as many slots as the pixels it visits, of 8 bytes, or
// of 18 where k_track_loop keeps its lists there too.
size_t track_list_bytes(int n) {
    const int g = track_cluster_grid(n);
    const int iters = (n + g * 256 - 1) / (g * 256);
    return (size_t)g * iters * 256 * (track_list_global(n) ? 18 : sizeof(int2));
}

// Compensated FP32 (the precision form's reduction).  two_sum is Knuth's
// error-free sum (s + e == a + b exactly); pair_add adds two (hi, lo) pairs
// with the rounding error of the high parts carried into the low part and
// the result renormalised (Dekker's fast two-sum), so a sum of many block
// sums keeps about twice the float precision.
__device__ __forceinline__ float2 two_sum(float a, float b) {
    const float s = __fadd_rn(a, b);
    const float bb = __fsub_rn(s, a);
    const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
    return make_float2(s, e);
}

__device__ __forceinline__ float2 pair_add(float2 x, float2 y) {
    const float2 s = two_sum(x.x, y.x);
    const float lo = __fadd_rn(__fadd_rn(x.y, y.y), s.y);
    const float hi = __fadd_rn(s.x, lo);
    return make_float2(hi, __fsub_rn(lo, __fsub_rn(hi, s.x)));
}

// Staging of the tracker state for the solve of one iteration.
struct SolveIO {
    double delta[16], last_pose[16], init_pose[16], pose[16];
    DevPose cur;
    float icp_error, icp_count, rgb_error, rgb_count;
    int failed;    // this iteration failed: pose rolled back to last_pose
    int updated;   // delta, pose and cur hold a Gauss-Newton update
};

// The acceptance test of the last iteration (Tracking.cc:398-408), one thread.
__device__ __noinline__ bool accept_pose(const SolveIO& io) {
    double pinv[16], p[16];
    mat4_rigid_inv(io.init_pose, pinv);
    mat4_mul(pinv, io.pose, p);
    const double tn = sqrt(p[3] * p[3] + p[7] * p[7] + p[11] * p[11]);
    return io.icp_error < 0.0001f && euler_sin_norm(p) <= 0.1 && tn <= 0.1;
}

// Shared scratch of solve_block.
struct SolveTmp {
    double W[9], V[9], T[16], dinv[16];
    double delta[16], pose[16];
    DevPose cur;
};

// The count and error tests of one iteration (Tracking.cc:319-360), one thread.
__device__ __forceinline__ void solve_checks(SolveIO& io, const double* s, int min_count) {
    const float r1 = (float)s[32 + 28];
    const float rgb_err = sqrtf((float)s[32 + 27]) / r1;
    io.rgb_error = rgb_err;
    io.rgb_count = r1;
    bool fail = isnan(rgb_err) || (int)r1 < min_count;
    if (!fail) {
        const float q1 = (float)s[28];
        const float icp_err = sqrtf((float)s[27]) / q1;
        io.icp_error = icp_err;
        io.icp_count = q1;
        fail = isnan(icp_err) || (int)q1 < min_count;
    }
    io.failed = fail ? 1 : 0;
    io.updated = fail ? 0 : 1;
}

// The Gauss-Newton step (Tracking.cc:361-394) from the FP64 sums s (ICP in
// s[0..28], RGB in s[32..60]): tmp.delta, pose and cur from io.delta and
// io.last_pose.
//
// One warp; every value is computed by the operations, in the order, of the
// plain one-thread form (LDL^T without pivoting -- the normal matrix is
// positive definite --, substitution, Sophus::SE3d::exp from the mathematics,
// two 4x4 products).  It is a chain of dependent FP64 operations between two
// iterations: one thread took 1.8 us (3.1 us where its spills met the pixel
// passes' registers).  Row i of the factorisation is lane i's (all lanes
// follow the divisions), the elements of the small matrices are one lane's
// each, sine and cosine come from one sincos (the same bits as sin and cos),
// and its three quotients from one division in three lanes.
__device__ __forceinline__ void solve_warp(const SolveIO& io, SolveTmp& tmp, const double* s) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    __syncwarp();
    // row `lane` of A = w RGB + ICP and of b
    const double w = (double)1e-4f;
    const int row = lane < 6 ? lane : 5;
    double a[6], yb;
#pragma unroll
    for (int j = 0; j < 6; ++j) {
        const int lo = min(row, j), hi = max(row, j);
        const int k = lo * 7 - lo * (lo - 1) / 2 + hi - lo;   // the sum of row[lo] row[hi]
        a[j] = s[32 + k] * w + s[k];
    }
    {
        const int k = row * 7 - row * (row - 1) / 2 + 6 - row;
        yb = s[32 + k] * w + s[k];
    }
    // (other rows' L are fetched where they are used: few live registers, as
    // spills on this chain cost more than the shuffles)
    double L[6], D[6], x[6], Dinv = 0;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        double t = a[k];
#pragma unroll
        for (int j = 0; j < k; ++j) t -= L[j] * __shfl_sync(full, L[j], k) * D[j];
        D[k] = __shfl_sync(full, t, k);
        const double inv = 1.0 / D[k];
        if (lane == k) Dinv = inv;
        L[k] = t * inv;
        const double yk = __shfl_sync(full, yb, k);
        if (lane > k) yb -= L[k] * yk;
    }
    yb *= Dinv;
#pragma unroll
    for (int i = 5; i >= 0; --i) {
        double t = __shfl_sync(full, yb, i);
#pragma unroll
        for (int j = i + 1; j < 6; ++j) t -= __shfl_sync(full, L[i], j) * x[j];
        x[i] = t;
    }
    // se3_exp of (upsilon, omega) = x: Rodrigues rotation and left Jacobian,
    // Taylor series near zero; lane 3 i + j holds element (i, j)
    const double th2 = x[3] * x[3] + x[4] * x[4] + x[5] * x[5];
    double ca, cb, cc;
    const double th = sqrt(th2);
    if (th < 1e-5) {
        ca = 1 - th2 / 6 + th2 * th2 / 120;
        cb = 0.5 - th2 / 24 + th2 * th2 / 720;
        cc = 1.0 / 6 - th2 / 120 + th2 * th2 / 5040;
    } else {
        double sn, co;
        sincos(th, &sn, &co);
        const double num = lane == 0 ? sn : lane == 1 ? 1 - co : th - sn;
        const double den = lane == 0 ? th : lane == 1 ? th2 : th2 * th;
        const double q = num / den;
        ca = __shfl_sync(full, q, 0);
        cb = __shfl_sync(full, q, 1);
        cc = __shfl_sync(full, q, 2);
    }
    const int i3 = lane / 3, j3 = lane - 3 * i3;
    if (lane < 9) {
        const int d = (j3 - i3 + 3) % 3;
        const int c = 3 - i3 - j3;   // the axis neither index names
        const double v = c == 0 ? x[3] : c == 1 ? x[4] : x[5];
        tmp.W[lane] = d == 0 ? 0.0 : d == 1 ? -v : v;
    }
    __syncwarp();
    if (lane < 9) {
        double w2 = 0;
#pragma unroll
        for (int k = 0; k < 3; ++k) w2 += tmp.W[i3 * 3 + k] * tmp.W[k * 3 + j3];
        const double I = i3 == j3 ? 1.0 : 0.0, wij = tmp.W[lane];
        tmp.T[i3 * 4 + j3] = I + ca * wij + cb * w2;
        tmp.V[lane] = I + cb * wij + cc * w2;   // the left Jacobian, for the translation
    }
    __syncwarp();
    if (lane < 3)
        tmp.T[lane * 4 + 3] = tmp.V[lane * 3] * x[0] + tmp.V[lane * 3 + 1] * x[1] + tmp.V[lane * 3 + 2] * x[2];
    else if (lane < 7)
        tmp.T[9 + lane] = lane == 6 ? 1.0 : 0.0;   // the last row
    __syncwarp();
    // delta = dT delta, pose = last delta^-1
    const int i4 = lane >> 2, j4 = lane & 3;
    double v = 0;
    if (lane < 16)
#pragma unroll
        for (int k = 0; k < 4; ++k) v += tmp.T[i4 * 4 + k] * io.delta[k * 4 + j4];
    if (lane < 16) tmp.delta[lane] = v;
    __syncwarp();
    if (lane < 16) {
        const double* d = tmp.delta;
        double o;
        if (i4 == 3)
            o = j4 == 3 ? 1.0 : 0.0;
        else if (j4 < 3)
            o = d[j4 * 4 + i4];
        else
            o = -(d[i4] * d[3] + d[4 + i4] * d[7] + d[8 + i4] * d[11]);
        tmp.dinv[lane] = o;
    }
    __syncwarp();
    if (lane < 16) {
        v = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) v += io.last_pose[i4 * 4 + k] * tmp.dinv[k * 4 + j4];
        tmp.pose[lane] = v;
        // the float view (make_dev_pose_d)
        float* c = (float*)&tmp.cur;
        if (i4 < 3) {
            if (j4 < 3) {
                c[i4 * 3 + j4] = (float)v;
                c[9 + j4 * 3 + i4] = (float)v;
            } else {
                c[18 + i4] = (float)v;
            }
        }
    }
}

// The Gauss-Newton update of one iteration and, after the last one, the
// acceptance test, on staged state by a whole block: io.delta / last_pose /
// init_pose / icp_error in; io.pose, delta, cur, errors, counts, failed and
// updated out (a failed count or error test leaves delta and cur as they were
// and sets pose = last_pose; a failed acceptance test does so after the
// update).  Ends with a block barrier.
// As a call, for k_track_loop: inlined, its FP64 state spills the passes' registers.
__device__ __noinline__ void solve_warp_call(const SolveIO& io, SolveTmp& tmp, const double* s) { solve_warp(io, tmp, s); }

template <bool kCall>
__device__ __forceinline__ void solve_block(SolveIO& io, SolveTmp& tmp, const double* s, int min_count, int is_final) {
    const int t = threadIdx.x;
    if (t < 32) {
        if constexpr (kCall)
            solve_warp_call(io, tmp, s);
        else
            solve_warp(io, tmp, s);
    } else if (t == 32)
        solve_checks(io, s, min_count);
    __syncthreads();
    const bool fail = io.failed != 0;
    if (t < 16) {
        io.pose[t] = fail ? io.last_pose[t] : tmp.pose[t];
        if (!fail) io.delta[t] = tmp.delta[t];
    } else if (t >= 32 && t < 32 + (int)(sizeof(DevPose) / 4)) {
        if (!fail) ((float*)&io.cur)[t - 32] = ((const float*)&tmp.cur)[t - 32];
    }
    __syncthreads();
    if (is_final && !fail) {
        if (t == 0 && !accept_pose(io)) {
            for (int i = 0; i < 16; ++i) io.pose[i] = io.last_pose[i];
            io.failed = 1;
        }
        __syncthreads();
    }
}

// The end of an iteration, in the block that finished last: the group sums
// of both passes in group order (FP64, or compensated FP32 in the precision
// form) -- value t & 63 (0..28 ICP, 32..60 RGB) over four fixed ranges of
// groups, then the ranges in order -- the Gauss-Newton update with one
// thread, and the new state written back in parallel.
template <bool kComp>
__device__ __forceinline__ void finish_iteration(TrackState* st, unsigned int* ticket, int NG, long long c,
                                                 long long q, float sigma, int min_count, int is_final,
                                                 SolveIO& io, double (&s_part)[4][64], float2 (&s_partc)[4][64],
                                                 double (&sums)[64]) {
    {
        const int val = threadIdx.x & 63, part = threadIdx.x >> 6;
        const int per = (NG + 3) / 4, g0 = part * per, g1 = min(NG, g0 + per);
        // the range's values are loaded 16 at a time before any is added (one
        // L2 round trip for the usual ten groups), then added in group order
        if constexpr (kComp) {
            // compensated FP32 over the groups; to FP64 only for the solve
            float2 t = make_float2(0.f, 0.f);
            if ((val & 31) < 29) {
                const float2* src = val < 32 ? &st->grp_icp2[0][val] : &st->grp_rgb2[0][val - 32];
                for (int g = g0; g < g1; g += 16) {
                    float2 v[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (g + j < g1) v[j] = __ldcg(src + (size_t)(g + j) * 32);
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (g + j < g1) t = pair_add(t, v[j]);
                }
            }
            s_partc[part][val] = t;
        } else {
            double t = 0;
            if ((val & 31) < 29) {
                const double* src = val < 32 ? &st->grp_icp[0][val] : &st->grp_rgb[0][val - 32];
                for (int g = g0; g < g1; g += 16) {
                    double v[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (g + j < g1) v[j] = __ldcg(src + (size_t)(g + j) * 32);
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (g + j < g1) t += v[j];
                }
            }
            s_part[part][val] = t;
        }
    }
    __syncthreads();
    if (threadIdx.x < 64) {
        if constexpr (kComp) {
            const float2 t = pair_add(pair_add(pair_add(s_partc[0][threadIdx.x], s_partc[1][threadIdx.x]),
                                               s_partc[2][threadIdx.x]),
                                      s_partc[3][threadIdx.x]);
            sums[threadIdx.x] = (double)t.x + (double)t.y;
        } else {
            sums[threadIdx.x] = ((s_part[0][threadIdx.x] + s_part[1][threadIdx.x]) + s_part[2][threadIdx.x]) +
                                s_part[3][threadIdx.x];
        }
    }
    __syncthreads();
    __shared__ SolveTmp tmp;
    solve_block<false>(io, tmp, sums, min_count, is_final);
    // write back in parallel
    if (threadIdx.x == 128) *ticket = 0;
    if (threadIdx.x < 16) {
        st->pose[threadIdx.x] = io.pose[threadIdx.x];
        if (io.updated) st->delta[threadIdx.x] = io.delta[threadIdx.x];
    } else if (threadIdx.x >= 32 && threadIdx.x < 32 + (int)(sizeof(DevPose) / 4)) {
        if (io.updated) ((float*)&st->cur)[threadIdx.x - 32] = ((const float*)&io.cur)[threadIdx.x - 32];
    } else if (threadIdx.x >= 64 && threadIdx.x < 93) {
        st->icp_sums[threadIdx.x - 64] = sums[threadIdx.x - 64];
        st->rgb_sums[threadIdx.x - 64] = sums[32 + threadIdx.x - 64];
    } else if (threadIdx.x == 96) {
        st->icp_error = io.icp_error;
        st->icp_count = io.icp_count;
        st->rgb_error = io.rgb_error;
        st->rgb_count = io.rgb_count;
        st->rgb_cnt = c;
        st->rgb_sq = q;
        st->sigma = sigma;
        st->failed = io.failed;
    }
}

// Shape of the group forms below: groups per block and resident blocks per
// SM (4: half the registers, some spilled; 2: none spilled).
constexpr int kGroupsPerBlock = 1;
constexpr int kGrpMinBlocks = 4;

// The passes for sessions sharing the GPU: one block per group does the work
// of the group's kTrackCluster logical blocks -- b = kTrackCluster * group + r
// in a grid of G blocks, r in rank order -- and adds their sums in rank order.
// A session's pass holds a quarter of the block slots for longer, and other
// sessions' passes run beside it.  A pass leaves its group sums in the
// tracker state; the last block of pass B to finish adds the groups and
// solves.
template <int kMinBlocks, bool kComp>
__device__ __forceinline__ void track_a_grp_body(const BlockCtx& ctx, TrackLevel L, TrackState* st, int2* list,
                                                 int* counts, int G, int gpc) {
    const int N = L.W * L.H, NG = G / kTrackCluster;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (st->failed) return;   // uniform over the grid: written by an earlier kernel
    __shared__ float sm[8 * 32];
    __shared__ long long smll[32];
    __shared__ double s_vals[kTrackCluster][32];
    __shared__ float s_f[kTrackCluster][32];
    __shared__ long long s_c[kTrackCluster][2];
    __shared__ PixelStage stg;
    const DevPose cur = st->cur, last = st->last;
    const int iters = (N + G * 256 - 1) / (G * 256);
    const unsigned lt = (1u << lane) - 1u;
    // thread 0 keeps the copies two chunks ahead of the block
    ChunkCursor prod{0, 0, 0, 0};
    uint32_t used = 0;
    if (threadIdx.x == 0) {
        mbar_init(&stg.bar[0], 1);
        mbar_init(&stg.bar[1], 1);
        prod.settle(ctx.bx, gpc, NG, iters, G * 256, N);
        for (int c = 0; c < 2 && prod.start >= 0; ++c) {
            stage_chunk(stg, c, L, prod.start, N);
            ++prod.k;
            prod.settle(ctx.bx, gpc, NG, iters, G * 256, N);
        }
    }
    __syncthreads();
    for (int j = 0; j < gpc; ++j) {
    const int g = ctx.bx * gpc + j;
    if (g >= NG) break;
    for (int r = 0; r < kTrackCluster; ++r) {
        const int b = g * kTrackCluster + r;
        int p = b * 256 + threadIdx.x;
        float acc[29];
#pragma unroll
        for (int k = 0; k < 29; ++k) acc[k] = 0.f;
        long long rc = 0, rsq = 0;
        const int gw = b * kTrackWarps + wid;
        int2* seg = list + (size_t)gw * iters * 32;
        int run = 0;
        for (int k = 0; k < iters; ++k, p += G * 256) {
            if (b * 256 + k * G * 256 >= N) break;   // uniform: no pixel of this chunk
            const int buf = (int)(used & 1u);
            if (!take_chunk(stg, buf, used >> 1)) {
                if (threadIdx.x == 0) atomicOr((unsigned*)&st->failed, 2u);
                return;
            }
            ++used;
            PixelIn in;
            if (p < N) in = staged_pixel(stg, buf, threadIdx.x);
            __syncthreads();   // buffer `buf` is read: the chunk two ahead may overwrite it
            if (threadIdx.x == 0 && prod.start >= 0) {
                stage_chunk(stg, buf, L, prod.start, N);
                ++prod.k;
                prod.settle(ctx.bx, gpc, NG, iters, G * 256, N);
            }
            int rr = -1;
            if (p < N) {
                float row[7];
                if (pixel_pass_a(L, cur, last, in, row, &rr)) add_products(row, acc);
                if (rr != -1) {
                    int d = (rr & 511) - 255;
                    rc += 1;
                    rsq += d * d;
                }
            }
            const unsigned m = __ballot_sync(0xffffffffu, rr != -1);
            if (rr != -1) seg[run + __popc(m & lt)] = make_int2(in.dxy, rr);
            run += __popc(m);
        }
        if (lane == 0) counts[gw] = run;
        const float bsum = block_sum29(acc, sm);
        const long long bc = __shfl_sync(0xffffffffu, block_sum_ll(rc, smll), 0);
        const long long bs = __shfl_sync(0xffffffffu, block_sum_ll(rsq, smll), 0);
        if constexpr (kComp) {
            if (wid == 0) s_f[r][lane] = lane < 29 ? bsum : 0.f;
            if (threadIdx.x == 0) {
                s_c[r][0] = bc;
                s_c[r][1] = bs;
            }
        } else {
            if (wid == 0)
                s_vals[r][lane] = lane < 29 ? (double)bsum : lane == 29 ? (double)bc : lane == 30 ? (double)bs : 0.0;
        }
        __syncthreads();   // sm / smll are reused by the next logical block
    }
    if (threadIdx.x < 31) {
        if constexpr (kComp) {
            if (threadIdx.x < 29) {
                float2 acc = make_float2(0.f, 0.f);
#pragma unroll
                for (int r = 0; r < kTrackCluster; ++r) acc = pair_add(acc, make_float2(s_f[r][threadIdx.x], 0.f));
                st->grp_icp2[g][threadIdx.x] = acc;
            } else {
                long long t = 0;
#pragma unroll
                for (int r = 0; r < kTrackCluster; ++r) t += s_c[r][threadIdx.x - 29];
                if (threadIdx.x == 29)
                    st->grp_cnt[g] = t;
                else
                    st->grp_sq[g] = t;
            }
        } else {
            double v = 0;
#pragma unroll
            for (int r = 0; r < kTrackCluster; ++r) v += s_vals[r][threadIdx.x];
            if (threadIdx.x < 29)
                st->grp_icp[g][threadIdx.x] = v;
            else if (threadIdx.x == 29)
                st->grp_cnt[g] = (long long)v;
            else
                st->grp_sq[g] = (long long)v;
        }
    }
    __syncthreads();   // s_vals / s_f / s_c are reused by the next group
    }
}

template <int kMinBlocks, bool kComp>
__device__ __forceinline__ void track_b_grp_body(const BlockCtx& ctx, TrackLevel L, TrackState* st,
                                                 unsigned int* ticket, const int2* list, const int* counts,
                                                 int seg_size, int min_count, int is_final, int NG, int gpc) {
    __shared__ float sm[32 * 29];
    __shared__ float s_rgb[kTrackCluster][32];
    __shared__ double s_part[4][64];
    __shared__ float2 s_partc[4][64];
    __shared__ double sums[64];
    __shared__ bool s_last;
    __shared__ SolveIO io;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    // stage the solve's inputs early (used by the last block)
    if (threadIdx.x >= 64 && threadIdx.x < 80) {
        const int i = threadIdx.x - 64;
        io.delta[i] = st->delta[i];
        io.last_pose[i] = st->last_pose[i];
        io.init_pose[i] = st->init_pose[i];
    }
    if (threadIdx.x == 80) {
        io.icp_error = st->icp_error;
        io.icp_count = st->icp_count;
    }
    if (st->failed) return;
    const DevPose cur = st->cur, last = st->last;
    // sigma = sqrt((float) sum / count) (Reduction.cu:606-608); every warp
    // adds the group counts itself (integers: exact in any order)
    long long c = 0, q = 0;
    for (int g = lane; g < NG; g += 32) {
        c += __ldcg(&st->grp_cnt[g]);
        q += __ldcg(&st->grp_sq[g]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        c += __shfl_xor_sync(0xffffffffu, c, o);
        q += __shfl_xor_sync(0xffffffffu, q, o);
    }
    const float sigma = sqrtf((float)q / (float)(c == 0 ? 1 : c));
    for (int j = 0; j < gpc; ++j) {
    const int grp = ctx.bx * gpc + j;
    if (grp >= NG) break;
    for (int r = 0; r < kTrackCluster; ++r) {
        const int b = grp * kTrackCluster + r;
        float acc[29];
#pragma unroll
        for (int k = 0; k < 29; ++k) acc[k] = 0.f;
        const int gw = b * kTrackWarps + wid;
        add_segment_rows(L, cur, last, sigma, list + (size_t)gw * seg_size, counts[gw], lane, acc);
        const float bsum = block_sum29(acc, sm);
        if (wid == 0) s_rgb[r][lane] = lane < 29 ? bsum : 0.f;
        __syncthreads();   // sm is reused by the next logical block
    }
    if constexpr (kComp) {
        if (threadIdx.x < 29) {
            float2 acc = make_float2(0.f, 0.f);
#pragma unroll
            for (int r = 0; r < kTrackCluster; ++r) acc = pair_add(acc, make_float2(s_rgb[r][threadIdx.x], 0.f));
            st->grp_rgb2[grp][threadIdx.x] = acc;
        }
    } else {
        if (threadIdx.x < 29) {
            double v = 0;
#pragma unroll
            for (int r = 0; r < kTrackCluster; ++r) v += (double)s_rgb[r][threadIdx.x];
            st->grp_rgb[grp][threadIdx.x] = v;
        }
    }
    __syncthreads();   // s_rgb is reused by the next group
    }
    // last block to finish
    __syncthreads();
    if (threadIdx.x == 0) s_last = ticket_acq_rel(ticket) == (unsigned)ctx.gx - 1u;
    __syncthreads();
    if (!s_last) return;
    finish_iteration<kComp>(st, ticket, NG, c, q, sigma, min_count, is_final, io, s_part, s_partc, sums);
}

template <int kMinBlocks, bool kComp>
__global__ void __launch_bounds__(256, kMinBlocks)
    k_track_a_grp(TrackLevel L, TrackState* st, int2* list, int* counts, int G, int gpc) {
    track_a_grp_body<kMinBlocks, kComp>(own_ctx(), L, st, list, counts, G, gpc);
}
template <int kMinBlocks, bool kComp>
__global__ void __launch_bounds__(256, kMinBlocks)
    k_track_a_grp_fused(const __grid_constant__ FusedParams<ArgsOf<decltype(&k_track_a_grp<kMinBlocks, kComp>)>> fp) {
    run_part(fp, [](const BlockCtx& c, const auto&... a) { track_a_grp_body<kMinBlocks, kComp>(c, a...); });
}

template <int kMinBlocks, bool kComp>
__global__ void __launch_bounds__(256, kMinBlocks)
    k_track_b_grp(TrackLevel L, TrackState* st, unsigned int* ticket, const int2* list, const int* counts,
                  int seg_size, int min_count, int is_final, int NG, int gpc) {
    track_b_grp_body<kMinBlocks, kComp>(own_ctx(), L, st, ticket, list, counts, seg_size, min_count, is_final, NG,
                                        gpc);
}
template <int kMinBlocks, bool kComp>
__global__ void __launch_bounds__(256, kMinBlocks)
    k_track_b_grp_fused(const __grid_constant__ FusedParams<ArgsOf<decltype(&k_track_b_grp<kMinBlocks, kComp>)>> fp) {
    run_part(fp, [](const BlockCtx& c, const auto&... a) { track_b_grp_body<kMinBlocks, kComp>(c, a...); });
}

// ------------------------------------------- the whole loop in one launch
//
// A session alone runs all its Gauss-Newton iterations in this one kernel: a
// cooperative grid of clusters, resident together, whose blocks hand each
// other their results through global memory instead of ending.  What bounds
// it is the chain of an iteration.  As two launches per iteration (clusters
// of the same shape: two launches, two state loads, two staging waits, four
// cluster barriers, a ticket) an iteration took 13 us on 160x120 pixels, 18
// on 320x240 and 26 on 640x480; here 8.7, 11.8 and 19 (a frame's 18
// iterations: 234 -> 154 us at 160x120, 393 -> 299 us at 640x480).  Per
// iteration:
//   - every block waits for the pose (8 slots), runs pass A over its pixels,
//     publishes its correspondence count and squared differences, reduces and
//     publishes its ICP sums while the other blocks' counts arrive;
//   - every block adds all counts (integers: exact), hence sigma, and runs
//     pass B from its correspondence list in shared memory (the gathered last
//     vertex is kept there by pass A) and publishes its RGB sums;
//   - the four blocks of cluster 0 each add one of the four group ranges of
//     both passes, block 0 adds the ranges, solves and publishes the pose.
// Pixels, lists, block sums, and the order in which they are added are those
// of the group kernels' logical grid of G blocks: the same bits.
//
// The exchanged values travel in 16-byte slots {3 words, epoch} stored and
// loaded as one 128-bit access each, so a slot that holds the expected epoch
// holds its data: no fences, tickets or second round trips.  A slot is
// rewritten only after everyone who needs its last value has published
// something that the rewriting waits for.  Every wait is bounded (kWaitPolls;
// for counts and sums LoopArgs::polls); a wait that gives up fails the frame (failed bit 1, reported by
// k_commit as kErrTimeout with the last pose) and its block leaves.
// The blocks must be resident together, hence the cooperative launch and the
// size rule of launch_track_loop.
constexpr int kLoopRows = 80;                       // blocks of one group range, at most
constexpr int kLoopMaxBuf = 12;
constexpr int kLoopScratch = kLoopRows / kTrackCluster * 32 * 8 + kLoopRows * 30 * 4;   // cluster 0's sums (14720)
constexpr int kLoopListBytes = 256 * (16 + 2);      // correspondence list of one chunk

// One 256-pixel chunk of the current frame (as PixelStage).
struct LoopStage {
    float4 v[256];
    float4 n[256];
    int16_t dx[256];
    int16_t dy[256];
    uint8_t ok[256];
    uint8_t g[256];
};

struct LoopArgs {
    TrackLevel L[3];
    int iters[3], min_count[3], G[3];
    int polls;     // loads of a count or sum before its wait gives up
    int nbuf;      // chunk buffers
    int chunks;    // chunks of a block, at most (the list's capacity)
    unsigned char* list;   // the lists in global memory (kGlobalList)
};

__device__ __forceinline__ void slot_put(TrackSlot* p, uint32_t x, uint32_t y, uint32_t z, uint32_t e) {
    asm volatile(
        "{\n"
        ".reg .b64 a, b;\n"
        ".reg .b128 t;\n"
        "mov.b64 a, {%1, %2};\n"
        "mov.b64 b, {%3, %4};\n"
        "mov.b128 t, {a, b};\n"
        "st.relaxed.gpu.global.b128 [%0], t;\n"
        "}\n" ::"l"(p), "r"(x), "r"(y), "r"(z), "r"(e)
        : "memory");
}

__device__ __forceinline__ uint4 slot_get(const TrackSlot* p) {
    uint4 v;
    asm volatile(
        "{\n"
        ".reg .b64 a, b;\n"
        ".reg .b128 t;\n"
        "ld.relaxed.gpu.global.b128 t, [%4];\n"
        "mov.b128 {a, b}, t;\n"
        "mov.b64 {%0, %1}, a;\n"
        "mov.b64 {%2, %3}, b;\n"
        "}\n"
        : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
        : "l"(p)
        : "memory");
    return v;
}

// Waits until the slot holds exchange e; false after `polls` loads.
__device__ __forceinline__ bool slot_wait(const TrackSlot* p, uint32_t e, int polls, uint4& v) {
    for (int i = polls; i > 0; --i) {
        v = slot_get(p);
        if (v.w == e) return true;
    }
    return false;
}

// The 29 block sums (lane l of warp 0 holds value l) into ten slots.
__device__ __forceinline__ void publish_sums(TrackSlot* slots, float r, int lane, uint32_t e) {
    const int k = lane < 10 ? 3 * lane : 0;
    const float x = __shfl_sync(0xffffffffu, r, k), y = __shfl_sync(0xffffffffu, r, k + 1),
                z = __shfl_sync(0xffffffffu, r, k + 2);
    if (lane < 10) slot_put(slots + lane, __float_as_uint(x), __float_as_uint(y), __float_as_uint(z), e);
}

// One lane: copy the chunk of pixels [start, min(start + 256, N)) into buf.
__device__ __forceinline__ void loop_fill(LoopStage& S, uint64_t* bar, const TrackLevel& L, int start, int N) {
    const int cnt = min(256, N - start);
    const uint32_t b16 = (uint32_t)cnt * 16u, b1 = ((uint32_t)cnt + 15u) & ~15u;
    const uint32_t b2 = ((uint32_t)cnt * 2u + 15u) & ~15u;
    mbar_arrive_expect_tx(bar, 2u * b16 + 2u * b2 + 2u * b1);
    bulk_copy_g2s(S.v, L.vcurr + start, b16, bar);
    bulk_copy_g2s(S.n, L.ncurr + start, b16, bar);
    bulk_copy_g2s(S.dx, L.dx + start, b2, bar);
    bulk_copy_g2s(S.dy, L.dy + start, b2, bar);
    bulk_copy_g2s(S.ok, L.rgbok + start, b1, bar);
    bulk_copy_g2s(S.g, L.gcurr + start, b1, bar);
}

// The sums of ng groups (kTrackCluster blocks each, from `src`: ten slots of
// one pass per block) in rank order, as FP64 (or compensated pairs) in
// ((double*)scratch)[group * 32 + value].  Whole block; false in a thread
// whose wait gave up.
template <bool kComp>
__device__ __forceinline__ bool range_sums(unsigned char* scratch, const TrackSlot* src, int ng, uint32_t e,
                                           int polls) {
    constexpr int kRowsAtOnce = 25;   // 25 x 10 slots by 250 threads
    const int t = threadIdx.x, nb = ng * kTrackCluster;
    float* const S = (float*)(scratch + kLoopRows / kTrackCluster * 32 * 8);
    bool ok = true;
    if (t < kRowsAtOnce * 10) {
        const int col = t % 10, row = t / 10;
        src += col;
        uint4 v[(kLoopRows + kRowsAtOnce - 1) / kRowsAtOnce];
#pragma unroll
        for (int j = 0; j < (kLoopRows + kRowsAtOnce - 1) / kRowsAtOnce; ++j)
            if (row + kRowsAtOnce * j < nb) v[j] = slot_get(src + (size_t)(row + kRowsAtOnce * j) * kSumSlots);
#pragma unroll
        for (int j = 0; j < (kLoopRows + kRowsAtOnce - 1) / kRowsAtOnce; ++j) {
            const int r = row + kRowsAtOnce * j;
            if (r < nb) {
                if (v[j].w != e) ok &= slot_wait(src + (size_t)r * kSumSlots, e, polls, v[j]);
                float* o = S + r * 30 + 3 * col;
                o[0] = __uint_as_float(v[j].x);
                o[1] = __uint_as_float(v[j].y);
                o[2] = __uint_as_float(v[j].z);
            }
        }
    }
    __syncthreads();
    const int val = t & 31;
    if (val < 29)
        for (int g = t >> 5; g < ng; g += kTrackWarps) {
            const float* x = S + kTrackCluster * g * 30 + val;
            if constexpr (kComp) {
                float2 v = make_float2(0.f, 0.f);
#pragma unroll
                for (int r = 0; r < kTrackCluster; ++r) v = pair_add(v, make_float2(x[30 * r], 0.f));
                ((float2*)scratch)[g * 32 + val] = v;
            } else {
                double v = 0;
#pragma unroll
                for (int r = 0; r < kTrackCluster; ++r) v += (double)x[30 * r];
                ((double*)scratch)[g * 32 + val] = v;
            }
        }
    __syncthreads();
    return ok;
}

template <bool kComp, bool kGlobalList>
__global__ void __cluster_dims__(kTrackCluster, 1, 1) __launch_bounds__(256, 2)
    k_track_loop(const __grid_constant__ LoopArgs A, TrackState* st, TrackSync* sync) {
    extern __shared__ __align__(128) unsigned char dyn[];
    __shared__ uint64_t bar[kLoopMaxBuf];
    __shared__ DevPose s_cur, s_last;
    __shared__ float sm[2][8 * 32];
    __shared__ uint32_t s_cnt[8], s_sq[8], s_tc[8];
    __shared__ unsigned long long s_tq[8];
    __shared__ double s_part[4][64];
    __shared__ double sums[64];
    __shared__ SolveIO io;
    __shared__ SolveTmp tmp;
    __shared__ int s_failed, s_bad;
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5, b = blockIdx.x;
    LoopStage* const stage = (LoopStage*)dyn;
    // this block's correspondence list: A.chunks * 256 entries of 16 bytes,
    // then of 2, a segment per warp
    unsigned char* const scratch = dyn + (size_t)A.nbuf * sizeof(LoopStage);
    unsigned char* const list = kGlobalList ? A.list + (size_t)b * A.chunks * kLoopListBytes : scratch;
    float4* const seg = (float4*)list + wid * A.chunks * 32;
    int16_t* const segd = (int16_t*)(list + (size_t)A.chunks * 256 * 16) + wid * A.chunks * 32;
    cg::cluster_group cl = cg::this_cluster();
    const unsigned base = sync->epoch, total = (unsigned)(A.iters[0] + A.iters[1] + A.iters[2]);
    if (t == 224)
        for (int i = 0; i < A.nbuf; ++i) mbar_init(&bar[i], 1);
    if (t == 0) s_failed = s_bad = 0;
    if (t < (int)(sizeof(DevPose) / 4)) {
        ((float*)&s_cur)[t] = ((const float*)&st->cur)[t];
        ((float*)&s_last)[t] = ((const float*)&st->last)[t];
        if (b == 0) ((float*)&io.cur)[t] = ((const float*)&st->cur)[t];
    }
    if (b == 0) {
        if (t >= 64 && t < 80) {
            io.delta[t - 64] = st->delta[t - 64];
            io.last_pose[t - 64] = st->last_pose[t - 64];
            io.init_pose[t - 64] = st->init_pose[t - 64];
        }
        if (t == 80) {
            io.icp_error = st->icp_error;
            io.icp_count = st->icp_count;
        }
    }
    __syncthreads();
    // chunks of this block at level l; copies of the first nbuf of them
    // (issued by one lane; every thread keeps the buffers' wait parities and
    // which of them have a copy in flight)
    auto chunks_of = [&](int l) {
        const int N = A.L[l].W * A.L[l].H, S = A.G[l] * 256;
        return b * 256 < N ? (N - b * 256 + S - 1) / S : 0;
    };
    uint32_t parity = 0, flight = 0;
    auto prefetch = [&](int l) {
        const int n = min(A.nbuf, chunks_of(l));
        if (t == 224) {
            fence_proxy_async_smem();
            for (int k = 0; k < n; ++k)
                loop_fill(stage[k], &bar[k], A.L[l], b * 256 + k * A.G[l] * 256, A.L[l].W * A.L[l].H);
        }
        flight |= (1u << n) - 1u;
    };
    unsigned e = base;
    bool fetched = false, alive = true;
    int bad = 0;
    const unsigned lt = (1u << lane) - 1u;
    for (int l = 2; l >= 0 && alive; --l) {
        const int iters = A.iters[l], G = A.G[l];
        if (iters == 0) continue;
        if (b >= G) {   // no pixels here at this level
            e += iters;
            continue;
        }
        if (!fetched) prefetch(l);
        fetched = true;
        int finer = l - 1;
        while (finer >= 0 && A.iters[finer] == 0) --finer;
        const TrackLevel& L = A.L[l];
        const int N = L.W * L.H, cb = chunks_of(l);
        const bool resident = cb <= A.nbuf;
        int f = 0;   // chunk fills taken at this level
        for (int it = 0; it < iters; ++it) {
            if (e != base && b != 0) {
                if (wid == 0) {
                    // a frame that failed at a coarser level, where this block
                    // had no pixels, says so under an earlier number (the limit
                    // is constant here: a variable one spills)
                    uint4 v;
                    bool got = false;
                    for (int i = 0; i < kWaitPolls && !got; ++i) {
                        v = slot_get(&sync->pose[b % kPoseCopies][lane & 7]);
                        const bool lost = (lane & 7) == 7 && v.x != 0 && v.w - base - 1u < total;
                        if (__any_sync(0xffffffffu, lost)) {
                            if (lane == 0) s_failed = 1;
                            got = true;
                            v.w = base;   // no pose
                        } else {
                            got = __all_sync(0xffffffffu, v.w == e);
                        }
                    }
                    if (!got) {
                        if (lane == 0) {
                            atomicOr((unsigned*)&st->failed, 2u);
                            s_failed = 2;
                        }
                    } else if (lane < 7 && v.w == e) {
                        uint32_t* c = (uint32_t*)&s_cur + 3 * lane;
                        c[0] = v.x;
                        c[1] = v.y;
                        c[2] = v.z;
                    }
                }
            }
            __syncthreads();   // (block 0 wrote its pose itself)
            if (s_failed) {
                alive = false;
                break;
            }
            const DevPose &cur = s_cur, &last = s_last;
            float acc[29];
#pragma unroll
            for (int k = 0; k < 29; ++k) acc[k] = 0.f;
            // pass A
            uint32_t rc = 0, rsq = 0;
            int run = 0;
            for (int k = 0; k < cb; ++k) {
                int buf = k;
                if (!resident) buf = f % A.nbuf;
                if (!resident || it == 0) {
                    if (!mbar_wait(&bar[buf], (parity >> buf) & 1u)) bad = 1;
                    parity ^= 1u << buf;
                    flight &= ~(1u << buf);
                }
                const int p = b * 256 + k * G * 256 + t;
                PixelIn in;
                if (p < N) {
                    const LoopStage& S = stage[buf];
                    in.vc = S.v[t];
                    const float4 n = S.n[t];
                    in.nc = make_float3(n.x, n.y, n.z);
                    in.ok = S.ok[t];
                    in.gc = S.g[t];
                    in.dxy = (int)(uint16_t)S.dx[t] | ((int)S.dy[t] << 16);
                }
                if (!resident) {
                    __syncthreads();   // the buffer is read: it may be filled again
                    if (f + A.nbuf < iters * cb) {
                        if (t == 224) {
                            fence_proxy_async_smem();
                            loop_fill(stage[buf], &bar[buf], L, b * 256 + (f + A.nbuf) % cb * G * 256, N);
                        }
                        flight |= 1u << buf;
                    }
                    ++f;
                }
                int r = -1;
                f3 vl;
                if (p < N) {
                    float row[7];
                    if (pixel_pass_a(L, cur, last, in, row, &r, &vl)) add_products(row, acc);
                }
                const int d = (r & 511) - 255;
                if (r != -1) {
                    rc += 1;
                    rsq += (uint32_t)(d * d);
                }
                const unsigned m = __ballot_sync(0xffffffffu, r != -1);
                if (r != -1) {
                    const int o = run + __popc(m & lt);
                    seg[o] = make_float4(vl.x, vl.y, vl.z, __int_as_float(in.dxy));
                    segd[o] = (int16_t)d;
                }
                run += __popc(m);
            }
            rc = __reduce_add_sync(0xffffffffu, rc);
            rsq = __reduce_add_sync(0xffffffffu, rsq);
            if (lane == 0) {
                s_cnt[wid] = rc;
                s_sq[wid] = rsq;
            }
            __syncthreads();
            if (t == 0) {
                uint32_t c = 0, q = 0;
#pragma unroll
                for (int w = 0; w < kTrackWarps; ++w) {
                    c += s_cnt[w];
                    q += s_sq[w];
                }
                slot_put(&sync->count[b], c, q, 0, e + 1);
            }
            if (it == iters - 1 && finer >= 0) prefetch(finer);   // its copies land during the rest of this iteration
            float bsum = block_sum29(acc, sm[0]);
            if (wid == 0) publish_sums(sync->sums[b], bsum, lane, e + 1);
            __syncwarp();   // the list is read by other lanes than wrote it
            // the first photometric row up to its weight, while the counts arrive
            RgbDir d0{};
            int diff0 = 0;
            if (lane < run) {
                const float4 v = seg[lane];
                const int dxy = __float_as_int(v.w);
                d0 = rgb_dir(xyz(v), (int)(int16_t)(dxy & 0xffff), dxy >> 16, L, cur, last);
                diff0 = segd[lane];
            }
            // sigma = sqrt((float) sum / count) (Reduction.cu:606-608)
            uint32_t tc = 0, tq = 0;   // at most three blocks' sums per thread: below 2^32
            for (int j = t; j < G; j += 256) {
                uint4 v;
                if (!slot_wait(&sync->count[j], e + 1, A.polls, v)) {
                    bad = 1;
                    continue;
                }
                tc += v.x;
                tq += v.y;
            }
            tc = __reduce_add_sync(0xffffffffu, tc);
            const uint32_t qlo = __reduce_add_sync(0xffffffffu, tq & 0xffffu);
            const uint32_t qhi = __reduce_add_sync(0xffffffffu, tq >> 16);
            if (lane == 0) {
                s_tc[wid] = tc;
                s_tq[wid] = ((unsigned long long)qhi << 16) + qlo;
            }
            bad = __syncthreads_or(bad);
            long long C = 0, Q = 0;
#pragma unroll
            for (int w = 0; w < kTrackWarps; ++w) {
                C += s_tc[w];
                Q += (long long)s_tq[w];
            }
            if (bad && b >= kTrackCluster) {
                if (t == 0) atomicOr((unsigned*)&st->failed, 2u);
                alive = false;
                break;
            }
            const float sigma = sqrtf((float)Q / (float)(C == 0 ? 1 : C));
            // pass B
#pragma unroll
            for (int k = 0; k < 29; ++k) acc[k] = 0.f;
            if (lane < run) {
                float row[7];
                rgb_weighted(d0, diff0, sigma, row);
                add_products(row, acc);
            }
            for (int i = lane + 32; i < run; i += 32) {
                const float4 v = seg[i];
                const int dxy = __float_as_int(v.w);
                float row[7];
                rgb_weighted(rgb_dir(xyz(v), (int)(int16_t)(dxy & 0xffff), dxy >> 16, L, cur, last), segd[i], sigma, row);
                add_products(row, acc);
            }
            bsum = block_sum29(acc, sm[1]);
            ++e;
            if (wid == 0) publish_sums(sync->sums[b] + 10, bsum, lane, e);
            const bool is_final = finer < 0 && it == iters - 1;
            if (b >= kTrackCluster) {
                if (is_final) alive = false;
                continue;
            }
            // cluster 0: block r adds group range r of both passes (the
            // ranges, and the orders inside, of finish_iteration); its list
            // space is free (block_sum29's barrier) and takes the sums.  The
            // ICP sums have arrived and are added while the last RGB sums come.
            const int NG = G / kTrackCluster, per = (NG + 3) / 4, g0 = b * per;
            const int ng = max(0, min(NG, g0 + per) - g0);
            for (int pass = 0; pass < 2; ++pass) {
                bad |= !range_sums<kComp>(scratch, &sync->sums[g0 * kTrackCluster][10 * pass], ng, e, A.polls);
                if (t < 32) {
                    double* dst = (double*)cl.map_shared_rank(&s_part[0][0], 0) + b * 64 + 32 * pass + t;
                    if constexpr (kComp) {
                        float2 v = make_float2(0.f, 0.f);
                        if (t < 29)
                            for (int g = 0; g < ng; ++g) v = pair_add(v, ((const float2*)scratch)[g * 32 + t]);
                        *(float2*)dst = v;
                    } else {
                        double v = 0;
                        if (t < 29)
#pragma unroll 4
                            for (int g = 0; g < ng; ++g) v += ((const double*)scratch)[g * 32 + t];
                        *dst = v;
                    }
                }
                __syncthreads();   // the scratch is read
            }
            bad = __syncthreads_or(bad);
            if (t == 0 && bad) *cl.map_shared_rank(&s_bad, 0) = 1;
            cl.sync();
            if (b != 0) {
                if (is_final) alive = false;
                continue;
            }
            if (t < 64) {
                if constexpr (kComp) {
                    const float2 v = pair_add(pair_add(pair_add(*(float2*)&s_part[0][t], *(float2*)&s_part[1][t]),
                                                       *(float2*)&s_part[2][t]),
                                              *(float2*)&s_part[3][t]);
                    sums[t] = (double)v.x + (double)v.y;
                } else {
                    sums[t] = ((s_part[0][t] + s_part[1][t]) + s_part[2][t]) + s_part[3][t];
                }
            }
            __syncthreads();
            solve_block<true>(io, tmp, sums, A.min_count[l], is_final ? 1 : 0);
            const int failed = s_bad ? 3 : io.failed;
            if (!is_final && t < 8 * kPoseCopies) {
                const int k = t & 7;
                const uint32_t* c = (const uint32_t*)&io.cur + 3 * k;
                if (k < 7)
                    slot_put(&sync->pose[t >> 3][k], c[0], c[1], c[2], e);
                else
                    slot_put(&sync->pose[t >> 3][7], (uint32_t)failed, 0, 0, e);
            }
            if (t >= 64 && t < 64 + (int)(sizeof(DevPose) / 4)) ((float*)&s_cur)[t - 64] = ((const float*)&io.cur)[t - 64];
            if (is_final || failed) {
                if (t < 16) {
                    st->pose[t] = io.pose[t];
                    st->delta[t] = io.delta[t];
                } else if (t >= 32 && t < 32 + (int)(sizeof(DevPose) / 4)) {
                    ((float*)&st->cur)[t - 32] = ((const float*)&io.cur)[t - 32];
                } else if (t >= 64 && t < 93) {
                    st->icp_sums[t - 64] = sums[t - 64];
                    st->rgb_sums[t - 64] = sums[32 + t - 64];
                } else if (t == 96) {
                    st->icp_error = io.icp_error;
                    st->icp_count = io.icp_count;
                    st->rgb_error = io.rgb_error;
                    st->rgb_count = io.rgb_count;
                    st->rgb_cnt = C;
                    st->rgb_sq = Q;
                    st->sigma = sigma;
                    st->failed = failed;
                }
                alive = false;
                break;
            }
        }
    }
    // copies still in flight (a frame that failed before a level it had
    // begun to stage) land before the block leaves
    while (flight) {
        const int i = __ffs((int)flight) - 1;
        mbar_wait(&bar[i], (parity >> i) & 1u);
        flight &= flight - 1u;
    }
}

// Single-step entry points (the reference's ICPStep / RGBStep): reduce the
// sums of one pass into out[29] (+ rgb count / sum of squares) in FP64.  Bound
// by latency: a block holds a few pixels a thread.  At 323x241 icp / rgb_a /
// rgb_b take 7.0 / 5.9 / 6.3 us; with one value after another through the
// block sum (145 shuffles a warp) and one thread adding the counts they took
// 10.4 / 17.0 / 10.3.
__global__ void __launch_bounds__(256) k_step_icp(TrackLevel L, DevPose cur, DevPose last, float* partials,
                                                  unsigned int* ticket, double* out) {
    __shared__ float sm[8 * 32];
    float acc[29];
#pragma unroll
    for (int k = 0; k < 29; ++k) acc[k] = 0.f;
    const int N = L.W * L.H;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < N; p += gridDim.x * blockDim.x) {
        const int y = p / L.W, x = p - y * L.W;
        float row[7];
        if (icp_row(L, cur, last, x, y, row)) add_products(row, acc);
    }
    const float bsum = block_tree29(acc, sm);
    if (threadIdx.x < 29) partials[(size_t)blockIdx.x * 32 + threadIdx.x] = bsum;
    if (!last_block(ticket)) return;
    __shared__ double scratch[8 * 32];
    __shared__ double sums[32];
    reduce_partials(partials, gridDim.x, 32, 29, sums, scratch);
    if (threadIdx.x < 29) out[threadIdx.x] = sums[threadIdx.x];
    if (threadIdx.x == 0) *ticket = 0;
}

__global__ void __launch_bounds__(256) k_step_rgb_a(TrackLevel L, DevPose cur, DevPose last, long long* partials,
                                                    unsigned int* ticket, int* residual, double* out) {
    __shared__ long long smll[32];
    long long rc = 0, rsq = 0;
    const int N = L.W * L.H;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < N; p += gridDim.x * blockDim.x) {
        const int y = p / L.W, x = p - y * L.W;
        int r = rgb_corresp(L, cur, last, x, y);
        residual[p] = r;
        if (r != -1) {
            int d = (r & 511) - 255;
            rc += 1;
            rsq += d * d;
        }
    }
    long long bc = block_sum_ll(rc, smll);
    long long bs = block_sum_ll(rsq, smll);
    if (threadIdx.x == 0) {
        partials[2 * blockIdx.x] = bc;
        partials[2 * blockIdx.x + 1] = bs;
    }
    if (!last_block(ticket)) return;
    // the blocks' counts, all threads together (integers: exact in any order;
    // one thread after another took 10 us)
    long long c = 0, q = 0;
    for (int b = threadIdx.x; b < gridDim.x; b += blockDim.x) {
        c += __ldcg(partials + 2 * b);
        q += __ldcg(partials + 2 * b + 1);
    }
    c = block_sum_ll(c, smll);
    q = block_sum_ll(q, smll);
    if (threadIdx.x == 0) {
        out[29] = (double)c;
        out[30] = (double)q;
        out[31] = sqrtf((float)q / (float)(c == 0 ? 1 : c));
        *ticket = 0;
    }
}

__global__ void __launch_bounds__(256) k_step_rgb_b(TrackLevel L, DevPose cur, DevPose last, float* partials,
                                                    unsigned int* ticket, const int* residual, double* out) {
    __shared__ float sm[8 * 32];
    const float sigma = (float)out[31];
    float acc[29];
#pragma unroll
    for (int k = 0; k < 29; ++k) acc[k] = 0.f;
    const int N = L.W * L.H;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < N; p += gridDim.x * blockDim.x) {
        int r = residual[p];
        if (r == -1) continue;
        const int y = p / L.W, x = p - y * L.W;
        float row[7];
        rgb_row(L, cur, last, x, y, r, sigma, row);
        add_products(row, acc);
    }
    const float bsum = block_tree29(acc, sm);
    if (threadIdx.x < 29) partials[(size_t)blockIdx.x * 32 + threadIdx.x] = bsum;
    if (!last_block(ticket)) return;
    __shared__ double scratch[8 * 32];
    __shared__ double sums[32];
    reduce_partials(partials, gridDim.x, 32, 29, sums, scratch);
    if (threadIdx.x < 29) out[threadIdx.x] = sums[threadIdx.x];
    if (threadIdx.x == 0) *ticket = 0;
}

// ---------------------------------------------------------------- launchers

// Two resident blocks of 256 threads per SM at most (the row kernels use
// ~110 registers per thread).
int track_grid(int n) {
    static int cap = 0;
    if (!cap) {
        int dev = 0, sms = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cap = sms > 0 ? 2 * sms : 296;
        if (cap > kTrackMaxBlocks) cap = kTrackMaxBlocks;
    }
    int g = (n + 255) / 256;
    return g < cap ? g : cap;
}

int launch_track_begin(TrackState* st, TrackSync* sync, const int iters[3], cudaStream_t s) {
    fb_launch(k_track_begin, (const void*)k_track_begin_fused, 1, 1, 0, s, st, sync, track_exchanges(iters));
    return 1;
}

// Chunks that a block of k_track_loop has at a level stay in shared memory
// for all of its iterations where they fit; a block with more than
// kLoopSmemChunks of them streams them through kLoopRing buffers every
// iteration, and keeps its list in global memory: both leave the L1 cache to
// the gathers (1280x960, 17 chunks: with the lists in shared memory 30 KB of
// L1 were left to 16 warps, and a level-0 iteration took 82 us instead of 65).
constexpr int kLoopSmemChunks = 6;
constexpr int kLoopRing = 3;
constexpr int kLoopMost = kLoopSmemChunks * ((int)sizeof(LoopStage) + kLoopListBytes);
static_assert(kLoopSmemChunks <= kLoopMaxBuf && kLoopMost >= kLoopSmemChunks * (int)sizeof(LoopStage) + kLoopScratch,
              "the list holds the scratch");

static const void* loop_kernel(bool compensated, bool global_list) {
    return compensated ? (global_list ? (const void*)k_track_loop<true, true> : (const void*)k_track_loop<true, false>)
                       : (global_list ? (const void*)k_track_loop<false, true>
                                      : (const void*)k_track_loop<false, false>);
}

// Clusters of k_track_loop resident at once on the current device with the
// most shared memory a launch takes (so the answer holds for every launch);
// -1 where it cannot run.
static int loop_clusters(bool compensated, bool global_list) {
    static std::mutex lock;
    static int resident[64][4] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
        cudaGetLastError();
        return -1;
    }
    std::lock_guard<std::mutex> guard(lock);
    int& r = resident[dev][(compensated ? 2 : 0) + (global_list ? 1 : 0)];
    if (!r) {
        const void* k = loop_kernel(compensated, global_list);
        r = -1;
        int coop = 0, n = 0;
        cudaLaunchConfig_t q = {};
        q.gridDim = dim3(kTrackMaxBlocks);
        q.blockDim = dim3(256);
        q.dynamicSmemBytes = kLoopMost;
        if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) == cudaSuccess && coop &&
            cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kLoopMost) == cudaSuccess &&
            cudaOccupancyMaxActiveClusters(&n, k, &q) == cudaSuccess && n > 0)
            r = n;
        cudaGetLastError();
    }
    return r;
}

// The logical grid of the tracking passes: track_grid rounded up to whole
// groups, at most as many as k_track_loop has clusters resident at once (a
// cluster needs all its blocks on one GPC, so fewer than 2 x SMs /
// kTrackCluster may fit).
int track_cluster_grid(int n) {
    static int cap = 0;
    if (!cap) {
        int dev = 0, sms = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        int c = sms > 0 ? 2 * sms / kTrackCluster : kTrackMaxGroups;
        const int r = loop_clusters(false, false);
        if (r > 0 && r < c) c = r;
        cudaGetLastError();
        if (c > kTrackMaxGroups) c = kTrackMaxGroups;
        cap = c * kTrackCluster;
    }
    const int g = (n + 255) / 256;
    const int gc = (g + kTrackCluster - 1) / kTrackCluster * kTrackCluster;
    return gc < cap ? gc : cap;
}

int launch_track_iter(const TrackLevel& L, TrackState* st, unsigned int* tickets, int2* residual, int* counts,
                      int min_count, bool is_final, cudaStream_t s, bool compensated) {
    const int n = L.W * L.H;
    const int g = track_cluster_grid(n);
    const int seg = (n + g * 256 - 1) / (g * 256) * 32;
    const int fin = is_final ? 1 : 0;
    const int ng = g / kTrackCluster, gpc = kGroupsPerBlock, gb = (ng + gpc - 1) / gpc;
    if (compensated) {
        fb_launch(k_track_a_grp<kGrpMinBlocks, true>, (const void*)k_track_a_grp_fused<kGrpMinBlocks, true>, gb, 256,
                  0, s, L, st, residual, counts, g, gpc);
        fb_launch(k_track_b_grp<kGrpMinBlocks, true>, (const void*)k_track_b_grp_fused<kGrpMinBlocks, true>, gb, 256,
                  0, s, L, st, tickets + 1, residual, counts, seg, min_count, fin, ng, gpc);
    } else {
        fb_launch(k_track_a_grp<kGrpMinBlocks, false>, (const void*)k_track_a_grp_fused<kGrpMinBlocks, false>, gb, 256,
                  0, s, L, st, residual, counts, g, gpc);
        fb_launch(k_track_b_grp<kGrpMinBlocks, false>, (const void*)k_track_b_grp_fused<kGrpMinBlocks, false>, gb, 256,
                  0, s, L, st, tickets + 1, residual, counts, seg, min_count, fin, ng, gpc);
    }
    return 2;
}

// Whether k_track_loop keeps its lists for n pixels in global memory.
bool track_list_global(int n) {
    const int g = track_cluster_grid(n);
    return (n + g * 256 - 1) / (g * 256) > kLoopSmemChunks;
}

// k_track_loop's launch for these levels, when its grid is resident at once.
int launch_track_loop(const TrackLevel lv[3], const int iters[3], const int min_count[3], TrackState* st,
                      TrackSync* sync, void* list, cudaStream_t s, bool compensated, int polls) {
    if (launch_recorder()) return 0;
    LoopArgs A{};
    A.polls = polls;
    int grid = 0, chunks = 0;
    bool global = false;
    for (int l = 0; l < 3; ++l) {
        A.L[l] = lv[l];
        A.iters[l] = iters[l];
        A.min_count[l] = min_count[l];
        const int n = lv[l].W * lv[l].H;
        A.G[l] = n > 0 ? track_cluster_grid(n) : 0;
        if (iters[l] <= 0) continue;
        if (n <= 0 || !lv[l].rgbok) return 0;
        grid = std::max(grid, A.G[l]);
        chunks = std::max(chunks, (n + A.G[l] * 256 - 1) / (A.G[l] * 256));
        global = global || track_list_global(n);
    }
    const int per = (grid / kTrackCluster + 3) / 4;
    if (grid == 0 || per * kTrackCluster > kLoopRows) return 0;
    A.chunks = chunks;
    A.nbuf = global ? kLoopRing : chunks;
    A.list = (unsigned char*)list;
    const int fixed = global ? kLoopScratch : std::max(chunks * kLoopListBytes, kLoopScratch);
    if (grid / kTrackCluster > loop_clusters(compensated, global)) return 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = (size_t)A.nbuf * sizeof(LoopStage) + fixed;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    void* args[] = {&A, &st, &sync};
    if (cudaLaunchKernelExC(&cfg, loop_kernel(compensated, global), args) == cudaSuccess) return 1;
    cudaGetLastError();
    return 0;
}

int launch_step_icp(const TrackLevel& L, const DevPose& cur, const DevPose& last, float* partials,
                     unsigned int* ticket, double* out, cudaStream_t s) {
    k_step_icp<<<track_grid(L.W * L.H), 256, 0, s>>>(L, cur, last, partials, ticket, out);
    return 1;
}

int launch_step_rgb(const TrackLevel& L, const DevPose& cur, const DevPose& last, float* partials,
                     unsigned int* tickets, int* residual, double* out, cudaStream_t s) {
    const int g = track_grid(L.W * L.H);
    k_step_rgb_a<<<g, 256, 0, s>>>(L, cur, last, (long long*)partials, tickets + 0, residual, out);
    k_step_rgb_b<<<g, 256, 0, s>>>(L, cur, last, partials, tickets + 1, residual, out);
    return 2;
}

}  // namespace fb
