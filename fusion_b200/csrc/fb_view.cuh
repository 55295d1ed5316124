// Device pieces that the visibility, z-range and integration kernels share.
#ifndef FB_VIEW_CUH
#define FB_VIEW_CUH

#include "fb_internal.h"

namespace fb {

// Fusion::CheckVertexVisibility / CheckBlockVisibility (FuseMap.cu:36-78);
// the eight corners are reached by the reference's sequence of float adds.
__device__ __forceinline__ bool vertex_visible(f3 p, const DevPose& P, const Intr& k, int W, int H,
                                               const MapGeom& g) {
    p = mv(P.Rinv, sub3(p, P.t));
    if (p.z < 1e-3f) return false;
    float u = fa(fd(fm(k.fx, p.x), p.z), k.cx), v = fa(fd(fm(k.fy, p.y), p.z), k.cy);
    return u >= 0 && v >= 0 && u < (float)W && v < (float)H && p.z >= g.depth_min && p.z <= g.depth_max;
}

__device__ __forceinline__ bool block_visible(int bx, int by, int bz, const DevPose& P, const Intr& k, int W, int H,
                              const MapGeom& g) {
    const float s = g.block_width;
    f3 c = mk3(fm((float)bx, s), fm((float)by, s), fm((float)bz, s));
    if (vertex_visible(c, P, k, W, H, g)) return true;
    c.z = fa(c.z, s);
    if (vertex_visible(c, P, k, W, H, g)) return true;
    c.y = fa(c.y, s);
    if (vertex_visible(c, P, k, W, H, g)) return true;
    c.x = fa(c.x, s);
    if (vertex_visible(c, P, k, W, H, g)) return true;
    c.z = fs(c.z, s);
    if (vertex_visible(c, P, k, W, H, g)) return true;
    c.y = fs(c.y, s);
    if (vertex_visible(c, P, k, W, H, g)) return true;
    c.x = fs(c.x, s);
    c.y = fa(c.y, s);
    if (vertex_visible(c, P, k, W, H, g)) return true;
    c.x = fa(c.x, s);
    c.y = fs(c.y, s);
    c.z = fa(c.z, s);
    if (vertex_visible(c, P, k, W, H, g)) return true;
    return false;
}

// Appends the warp's visible blocks to the list (one atomic per warp; every
// lane calls it).
__device__ __forceinline__ void append_visible(const MapView& m, bool vis, int slot, const HEntry& e) {
    unsigned mask = __ballot_sync(0xffffffffu, vis);
    if (mask) {
        int base = 0;
        const int lane = threadIdx.x & 31;
        if (lane == 0) base = atomicAdd(&m.ctr->n_visible, __popc(mask));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (vis) {
            int o = base + __popc(mask & ((1u << lane) - 1));
            if (o < m.NS) {
                m.visible[o] = slot;
                m.vis_blocks[o] = e;   // read by integration and z ranges without a second gather
            } else {
                atomicOr(&m.ctr->err, kErrVisibleFull);
            }
        }
    }
}

__device__ __forceinline__ void grow_box(int (&lo)[3], int (&hi)[3], const HEntry& e) {
    lo[0] = min(lo[0], (int)e.x);
    lo[1] = min(lo[1], (int)e.y);
    lo[2] = min(lo[2], (int)e.z);
    hi[0] = max(hi[0], (int)e.x);
    hi[1] = max(hi[1], (int)e.y);
    hi[2] = max(hi[2], (int)e.z);
}

// Widens the box of the visible blocks by the warp's bounds.
__device__ __forceinline__ void widen_box(const MapView& m, int (&lo)[3], int (&hi)[3]) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        lo[a] = __reduce_min_sync(0xffffffffu, lo[a]);
        hi[a] = __reduce_max_sync(0xffffffffu, hi[a]);
    }
    if ((threadIdx.x & 31) == 0 && lo[0] <= hi[0]) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            atomicMin(&m.ctr->bmin[a], lo[a]);
            atomicMax(&m.ctr->bmax[a], hi[a]);
        }
    }
}

// A visible block's rectangle in the z-range images and its depth interval
// (positive floats as integers).
struct ZRect {
    int x, y, w, cells;   // upper left cell, width, cells in all (at most 16 x 16)
    int zmin, zmax;
};

// Projection::projectBlock (RenderScene.cu:54-104) cut to the first tile (see
// raycast.cu); false when the block covers nothing.
__device__ __forceinline__ bool project_block(const MapView& m, const HEntry& e, const DevPose& P, const Intr& k,
                                              ZRect& r) {
    const int zc = m.zc, zr = m.zr;
    int ulx = zc, uly = zr, lrx = -1, lry = -1;
    float zx = m.g.depth_max, zy = m.g.depth_min;
    for (int c = 0; c < 8; ++c) {
        const int tx = e.x + ((c & 1) ? 1 : 0), ty = e.y + ((c & 2) ? 1 : 0), tz = e.z + ((c & 4) ? 1 : 0);
        f3 p = mk3(fm((float)(tx * 8), m.g.voxel_size), fm((float)(ty * 8), m.g.voxel_size),
                   fm((float)(tz * 8), m.g.voxel_size));
        p = mv(P.Rinv, sub3(p, P.t));
        if ((double)p.z < 2e-1) continue;
        const float qx = fd(fa(fd(fm(k.fx, p.x), p.z), k.cx), 8.0f);
        const float qy = fd(fa(fd(fm(k.fy, p.y), p.z), k.cy), 8.0f);
        // upperLeft / lowerRight are short2 (DeviceMap.h:11-18)
        if ((float)ulx > floorf(qx)) ulx = (short)(int)floorf(qx);
        if ((float)lrx < ceilf(qx)) lrx = (short)(int)ceilf(qx);
        if ((float)uly > floorf(qy)) uly = (short)(int)floorf(qy);
        if ((float)lry < ceilf(qy)) lry = (short)(int)ceilf(qy);
        if (zx > p.z) zx = p.z;
        if (zy < p.z) zy = p.z;
    }
    if (ulx < 0) ulx = 0;
    if (uly < 0) uly = 0;
    if (lrx >= zc) lrx = zc - 1;
    if (lry >= zr) lry = zr - 1;
    if (ulx > lrx || uly > lry) return false;
    if (zx < m.g.depth_min) zx = m.g.depth_min;
    if (zy < m.g.depth_min) return false;
    const int ex = min(ulx + 15, lrx), ey = min(uly + 15, lry);
    r.x = ulx;
    r.y = uly;
    r.w = ex - ulx + 1;
    r.cells = r.w * (ey - uly + 1);
    r.zmin = __float_as_int(zx);
    r.zmax = __float_as_int(zy);
    return true;
}

// A CTA's rectangles min/max-ed into the z-range images (fillBlocks,
// RenderScene.cu:156-179).  One block of kViewBatch per thread of two warps,
// then a rectangle per warp with a cell per lane: a thread filling its own
// rectangle sent every atomic of a warp to 32 places, from the few CTAs that
// the list fills (4200 blocks of 8 mm at 1280x960: 20 us for k_zrange).
constexpr int kViewBatch = 64;
struct ZRects {
    ZRect r[kViewBatch];
    int n;
};

// The warps of threads [0, kViewBatch) offer their rectangles.
__device__ __forceinline__ void add_rect(const MapView& m, ZRects& s, bool has, const ZRect& r) {
    const unsigned mask = __ballot_sync(0xffffffffu, has);
    const int lane = threadIdx.x & 31;
    int base = 0;
    if (lane == 0 && mask) {
        base = atomicAdd(&s.n, __popc(mask));
        atomicAdd(&m.ctr->n_tiles, __popc(mask));
    }
    base = __shfl_sync(0xffffffffu, base, 0);
    if (has) s.r[base + __popc(mask & ((1u << lane) - 1))] = r;
}

__device__ __forceinline__ void fill_rects(const MapView& m, const ZRects& s) {
    const int lane = threadIdx.x & 31;
    for (int q = threadIdx.x >> 5; q < s.n; q += blockDim.x >> 5) {
        const ZRect r = s.r[q];
        const unsigned inv = (65536u + (unsigned)r.w - 1u) / (unsigned)r.w;   // c / w = c inv >> 16 for c < 256, w <= 16
        for (int c = lane; c < r.cells; c += 32) {
            const int dy = (int)(((unsigned)c * inv) >> 16);
            const int cell = (r.y + dy) * m.zc + r.x + c - dy * r.w;
            atomicMin((int*)&m.zmin[cell], r.zmin);
            atomicMax((int*)&m.zmax[cell], r.zmax);
        }
    }
}

// The z-range images, the box and the counters before a z-range pass, by the
// threads of a grid.
__device__ __forceinline__ void zrange_clear(const MapView& m, int gtid, int gstride) {
    if (gtid < 3) {
        m.ctr->bmin[gtid] = 0x7fffffff;
        m.ctr->bmax[gtid] = -0x7fffffff;
    }
    if (gtid == 0) {
        m.ctr->ray_next = 0;
        m.ctr->n_tiles = 0;   // counted again by each z-range pass
    }
    const int n = m.zc * m.zr;
    for (int i = gtid; i < n; i += gstride) {
        m.zmin[i] = 100.f;   // CreateRenderingBlocks uploads 100 (RenderScene.cu:245-251)
        m.zmax[i] = 0.f;     // and clears zRangeY (RenderScene.cu:244)
    }
}

// The box of the dense block index from the z-range pass's bounds.
struct GridBox {
    int o[3], n[3];
    bool on;
};

__device__ __forceinline__ GridBox grid_box(const MapView& m) {
    const MapCounters* c = m.ctr;
    GridBox b;
    long long vol = 1;
    for (int a = 0; a < 3; ++a) {
        b.o[a] = c->bmin[a] - 1;
        b.n[a] = c->bmax[a] - c->bmin[a] + 3;
        if (b.n[a] < 1) b.n[a] = 0;
        vol *= b.n[a];
    }
    b.on = c->bmin[0] <= c->bmax[0] && vol > 0 && vol <= m.grid_cap;
    return b;
}

// Empties the dense block index over its box, by the threads of a grid (each
// derives the box; the first ones publish it for the fill and the raycast).
__device__ __forceinline__ void grid_clear(const MapView& m, int gtid, int gstride) {
    const GridBox gb = grid_box(m);
    if (gtid < 3) {
        m.ctr->g_o[gtid] = gb.o[gtid];
        m.ctr->g_n[gtid] = gb.on ? gb.n[gtid] : 0;
        if (gtid == 0) m.ctr->g_on = gb.on ? 1 : 0;
    }
    if (!gb.on) return;
    const int vol = gb.n[0] * gb.n[1] * gb.n[2];
    int4* g4 = (int4*)m.grid;
    const int4 none = make_int4(-1, -1, -1, -1);
    for (int i = gtid; i < (vol + 3) / 4; i += gstride) g4[i] = none;
}

}  // namespace fb

#endif
