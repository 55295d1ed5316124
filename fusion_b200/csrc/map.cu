// Voxel-block hash map: block allocation, visibility and TSDF/colour
// integration (the reference's Mapping/DeviceMap.cu, Mapping/FuseMap.cu).
//
// Allocation is deterministic.  The reference lets every pixel's probes race
// for a per-bucket try-lock (DeviceMap.cu:23-62): requests that lose the lock
// are dropped and entries can be duplicated.  Here one frame's requests are
// collected first and then inserted as if one at a time, without contention,
// in canonical order -- ascending (bucket, x, y, z) -- so the resulting hash
// state (slot, voxel block and chain link of every entry) depends only on the
// inputs.  The kernels:
//   requests : per pixel, the reference's probe walk along the truncation band
//              (Fusion::CreateBlocks, FuseMap.cu:80-111); blocks that are not in
//              the map go into a per-frame open-addressing request set (CAS on
//              64-bit keys); the first insert of a key appends it to the list
//              of new blocks, counts it in its bin of consecutive buckets and
//              chains it there.
//   insert   : each new block finds its canonical rank -- its bin's start plus
//              the blocks of the bin's chain before it -- and computes from
//              it alone where the sequential insertion would put it:
//              free-stack position, head slot or excess slot, and its chain
//              link; the one block per bucket that extends an existing chain
//              links the old tail.  The last block to finish writes the
//              counters after the frame and clears the bins.  If the pool or
//              the excess list would run out, or an earlier exhaustion left
//              empty entries inside chains, a single thread of that last
//              block performs the same insertions one by one with the
//              reference's exact CreateBlock rules instead.
// Visibility walks the list of allocated entries rather than every slot of
// the table (CheckVisibleBlockKernel, FuseMap.cu:113-138, scans all of them).
// Integration processes one visible block per CTA iteration: 256 threads, two
// voxels each, one 16-byte load (issued one block ahead) and at most one
// 16-byte store per thread; the per-pixel inputs come from the frame's fusion
// records (one 16-byte gather of depth and normal, one word of colour).
#include <cuda_fp16.h>

#include "fb_fused.cuh"
#include "fb_internal.h"
#include "fb_view.cuh"

namespace fb {

// Whether block (x, y, z) has a live entry (FindEntry, DeviceMap.cu:122-135);
// its bucket b, and he = the bucket's head slot is empty.
__device__ __forceinline__ bool find_entry(const MapView& m, int x, int y, int z, uint32_t b, bool& he) {
    HEntry e = m.entries[b];
    he = e.ptr == -1;
    if (!he && e.x == x && e.y == y && e.z == z) return true;
    for (int guard = 0; e.offset > 0 && e.offset <= m.NE && guard <= m.NE; ++guard) {
        e = m.entries[m.NB + e.offset - 1];
        if (e.x == x && e.y == y && e.z == z && e.ptr != -1) return true;
    }
    return false;
}

__device__ __forceinline__ unsigned long long block_key(int x, int y, int z) {
    return (1ull << 63) | ((unsigned long long)(x & 0xFFFF) << 32) | ((unsigned long long)(y & 0xFFFF) << 16) |
           (unsigned long long)(z & 0xFFFF);
}

__device__ __forceinline__ uint32_t mix64(unsigned long long k) {
    k ^= k >> 33;
    k *= 0xff51afd7ed558ccdull;
    k ^= k >> 33;
    k *= 0xc4ceb9fe1a85ec53ull;
    k ^= k >> 33;
    return (uint32_t)k;
}

__device__ __forceinline__ void request_block(const MapView& m, int x, int y, int z) {
    if (x < -kCoordLimit || x > kCoordLimit || y < -kCoordLimit || y > kCoordLimit || z < -kCoordLimit ||
        z > kCoordLimit) {
        atomicOr(&m.ctr->err, kErrCoordRange);
        return;
    }
    const uint32_t bucket = bucket_of_m(x, y, z, (uint32_t)m.NB, m.nb_mask);
    bool he;
    if (find_entry(m, x, y, z, bucket, he)) return;
    const unsigned long long key = block_key(x, y, z);
    uint32_t h = mix64(key) & (uint32_t)(m.reqcap - 1);
    for (int probe = 0; probe < 64; ++probe) {
        unsigned long long old = atomicCAS(&m.reqset[h], 0ull, key);
        if (old == 0ull) {
            int idx = atomicAdd(&m.ctr->n_req, 1);
            if (idx < m.newcap) {
                NewBlock nb;
                nb.x = (short)x;
                nb.y = (short)y;
                nb.z = (short)z;
                nb.he = he ? 1 : 0;
                nb.bucket = bucket;
                nb.setslot = (int)h;
                // one block of a bucket with an empty head fills it: which of
                // them is counted for it does not matter
                nb.fills = atomicAdd(&m.bucket_cnt[bucket], 1) == 0 && he ? 1 : 0;
                const uint32_t bin = bucket >> m.bin_shift;
                atomicAdd(&m.bins->cnt[bin], 1ull | (unsigned long long)nb.fills << 32);
                nb.next = atomicExch(&m.bins->head[bin], idx);
                nb.pad[0] = nb.pad[1] = 0;
                m.newblk[idx] = nb;
            } else {
                atomicOr(&m.ctr->err, kErrNewListFull);
                atomicExch(&m.reqset[h], 0ull);
            }
            return;
        }
        if (old == key) return;
        h = (h + 1) & (uint32_t)(m.reqcap - 1);
    }
    atomicOr(&m.ctr->err, kErrRequestSetFull);
}

// Fusion::CreateBlocks (FuseMap.cu:80-111) for one pixel of the raw depth map.
__device__ __forceinline__ void request_pixel(const MapView& m, const float* __restrict__ raw, int rp, int x, int y,
                                              const Intr& k, const DevPose* __restrict__ posep) {
    const float z = raw[(size_t)y * rp + x];
    const float dmin = m.g.depth_min, dmax = m.g.depth_max;
    if (isnan(z) || z < dmin || z > dmax) return;
    const DevPose P = *posep;
    const float thresh = m.g.trunc_dist / 2;
    const float zn = fminf(dmax, fs(z, thresh));
    const float zf = fminf(dmax, fa(z, thresh));
    if (zn >= zf) return;
    const float vinv = m.g.voxel_size_inv;
    const float ux = fs((float)x, k.cx), uy = fs((float)y, k.cy);
    f3 pn = mul3(add3(mv(P.R, mk3(fm(fm(zn, ux), k.invfx), fm(fm(zn, uy), k.invfy), zn)), P.t), vinv);
    f3 pf = mul3(add3(mv(P.R, mk3(fm(fm(zf, ux), k.invfx), fm(fm(zf, uy), k.invfy), zf)), P.t), vinv);
    f3 dir = sub3(pf, pn);
    const float len = norm3(dir);
    const int nSteps = (int)ceil(2.0 * (double)len);
    dir = div3(dir, (float)(nSteps - 1));
    int px = 0, py = 0, pz = 0;
    bool have = false;
    for (int i = 0; i < nSteps; ++i) {
        // make_int3(float3) truncates toward zero (VectorMath.h:36-38)
        int bx = block_of(__float2int_rz(pn.x)), by = block_of(__float2int_rz(pn.y)),
            bz = block_of(__float2int_rz(pn.z));
        if (!have || bx != px || by != py || bz != pz) {
            request_block(m, bx, by, bz);
            px = bx;
            py = by;
            pz = bz;
            have = true;
        }
        pn = add3(pn, dir);
    }
}

// The last of n blocks to come here (true in every thread of it): what the
// blocks wrote before is visible to it.  It resets the ticket.
__device__ __forceinline__ bool last_to_finish(unsigned* ticket, unsigned n) {
    __shared__ bool s_last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(ticket, 1u) == n - 1u;
        if (s_last) *ticket = 0;
        __threadfence();
    }
    __syncthreads();
    return s_last;
}

__device__ __forceinline__ void alloc_requests_body(const BlockCtx& ctx, MapView m, const float* __restrict__ raw,
                                                    int rp, int W, int H, Intr k, const DevPose* __restrict__ posep,
                                                    const int* __restrict__ skip) {
    if (skip && *skip) return;   // the whole grid
    const int x = ctx.bx * blockDim.x + threadIdx.x;
    const int y = ctx.by * blockDim.y + threadIdx.y;
    if (x < W && y < H) request_pixel(m, raw, rp, x, y, k, posep);
}

__global__ void __launch_bounds__(256) k_alloc_requests(MapView m, const float* __restrict__ raw, int rp, int W,
                                  int H, Intr k, const DevPose* __restrict__ posep, const int* __restrict__ skip) {
    alloc_requests_body(own_ctx(), m, raw, rp, W, H, k, posep, skip);
}
FB_FUSED_KERNEL(k_alloc_requests, alloc_requests_body, 256)

__device__ __forceinline__ bool coord_less(const NewBlock& a, const NewBlock& b) {
    if (a.x != b.x) return a.x < b.x;
    if (a.y != b.y) return a.y < b.y;
    return a.z < b.z;
}

// CreateBlock (DeviceMap.cu:23-62) without lock contention, one block at a
// time, for the sequential path.  Returns the slot written or -1.
__device__ int create_block_seq(const MapView& m, int x, int y, int z, int& hc, int& ep, int& holes) {
    const int b = (int)bucket_of_m(x, y, z, (uint32_t)m.NB, m.nb_mask);
    HEntry* e = &m.entries[b];
    HEntry* eEmpty = nullptr;
    if (e->x == x && e->y == y && e->z == z && e->ptr != -1) return -1;
    if (e->ptr == -1) eEmpty = e;
    for (int guard = 0; e->offset > 0 && e->offset <= m.NE && guard <= m.NE; ++guard) {
        e = &m.entries[m.NB + e->offset - 1];
        if (e->x == x && e->y == y && e->z == z && e->ptr != -1) return -1;
        if (e->ptr == -1 && !eEmpty) eEmpty = e;
    }
    // CreateEntry (DeviceMap.cu:12-21)
    auto create_entry = [&](int offset) {
        HEntry n;
        n.x = (short)x;
        n.y = (short)y;
        n.z = (short)z;
        n.pad = 0;
        int old = hc--;
        int ptr = old >= 0 ? m.heap[old] : -1;
        if (ptr != -1) {
            n.ptr = ptr;
            n.offset = offset;
        } else {
            n.ptr = -1;
            n.offset = 0;
        }
        return n;
    };
    if (eEmpty) {
        *eEmpty = create_entry(e->offset);
        if (eEmpty->ptr == -1) holes = 1;
        return (int)(eEmpty - m.entries);
    }
    int offset = ep++;
    if (offset <= m.NE) {
        HEntry* n = &m.entries[m.NB + offset - 1];
        *n = create_entry(0);
        e->offset = offset;
        if (n->ptr == -1) holes = 1;
        return (int)(n - m.entries);
    }
    return -1;
}

// Starts of the bins (blocks, blocks with `fills`) in shared memory: an
// exclusive scan of their counts by 256 threads, each a run of consecutive
// bins.  Returns all of them.
__device__ __forceinline__ int2 scan_bins(const MapView& m, int2* start) {
    constexpr int kEach = kAllocBins / 256;
    __shared__ int2 s_warp[8];
    const int t = threadIdx.x;
    const ulonglong2* src = reinterpret_cast<const ulonglong2*>(m.bins->cnt + t * kEach);
    int2 v[kEach];
    int2 sum = make_int2(0, 0);
#pragma unroll
    for (int q = 0; q < kEach / 2; ++q) {
        const ulonglong2 c = src[q];
        v[2 * q] = make_int2((int)(uint32_t)c.x, (int)(c.x >> 32));
        v[2 * q + 1] = make_int2((int)(uint32_t)c.y, (int)(c.y >> 32));
    }
#pragma unroll
    for (int q = 0; q < kEach; ++q) {
        sum.x += v[q].x;
        sum.y += v[q].y;
    }
    int2 run = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int ux = __shfl_up_sync(0xffffffffu, run.x, o), uy = __shfl_up_sync(0xffffffffu, run.y, o);
        if ((t & 31) >= o) {
            run.x += ux;
            run.y += uy;
        }
    }
    if ((t & 31) == 31) s_warp[t >> 5] = run;
    __syncthreads();
    run.x -= sum.x;
    run.y -= sum.y;
    int2 all = make_int2(0, 0);
#pragma unroll
    for (int w = 0; w < 8; ++w) {
        if (w < (t >> 5)) {
            run.x += s_warp[w].x;
            run.y += s_warp[w].y;
        }
        all.x += s_warp[w].x;
        all.y += s_warp[w].y;
    }
#pragma unroll
    for (int q = 0; q < kEach; ++q) {
        start[t * kEach + q] = run;
        run.x += v[q].x;
        run.y += v[q].y;
    }
    __syncthreads();
    return all;
}

// Where the sequential insertion in canonical order puts a new block, from
// its bin: rank = its place in the order, among = its place in its bucket,
// xbefore = blocks of the buckets before that go to the excess list, more =
// another of its bucket follows.
struct NewPlace {
    int rank, among, xbefore;
    bool more;
};

__device__ __forceinline__ NewPlace place_of(const MapView& m, const int2* starts, const NewBlock& nb, int M) {
    const uint32_t bin = nb.bucket >> m.bin_shift;
    const int2 start = starts[bin];
    int less = 0, fills = 0, among = 0, same = 0;
    int q = m.bins->head[bin];
    for (int guard = 0; q >= 0 && guard < M; ++guard) {
        const NewBlock o = m.newblk[q];
        q = o.next;
        if (o.bucket < nb.bucket) {
            ++less;
            fills += o.fills;
        } else if (o.bucket == nb.bucket) {
            ++same;
            among += coord_less(o, nb) ? 1 : 0;
        }
    }
    NewPlace p;
    p.rank = start.x + less + among;
    p.among = among;
    p.xbefore = start.x + less - (start.y + fills);
    p.more = among + 1 < same;
    return p;
}

// The insertion (parallel or sequential path), the clearing of the request
// set, of the per-bucket counters and, in the block that finishes last, of the
// bins for the next frame, and the map counters after this frame (written
// there too, when every block has read them).  zinit: the z-range images and
// counters of the pass that follows are cleared as well.
// It is bound by latency (counters, bins, chain, free stack, entry): 9 us at
// 640x480.  With the request kernel it replaces a counting sort over all
// buckets in five launches: 38 -> 20 us a frame at 640x480 with 2^20 buckets
// (19 us of it the two scans of the buckets), 22 -> 13 us at 160x120 with 2^18.
__device__ __forceinline__ void alloc_insert_body(const BlockCtx& ctx, MapView m, int zinit) {
    MapCounters* c = m.ctr;
    const int M = min(c->n_req, m.newcap);
    const int gtid = ctx.bx * blockDim.x + threadIdx.x, gstride = ctx.gx * blockDim.x;
    const int hc0 = c->heap_counter, ep0 = c->entry_ptr, na0 = c->n_alloc, holes0 = c->holes;
    if (zinit) zrange_clear(m, gtid, gstride);
    __shared__ int2 starts[kAllocBins];
    bool fast = true;
    if (ctx.bx * (int)blockDim.x < M) {   // the block has new blocks to insert
        const int2 all = scan_bins(m, starts);
        // blocks that do not fill a head slot go to the excess list
        const int excess = all.x - all.y;
        if (threadIdx.x == 0) c->excess_total = excess;   // the same from every block
        // the parallel path reproduces sequential insertion only while the
        // free stack and the excess list suffice and no chain holds an empty
        // entry left by an earlier exhaustion
        fast = M <= hc0 + 1 && ep0 - 1 + excess <= m.NE && !holes0;
    }
    for (int i = gtid; i < M; i += gstride) {
        const NewBlock nb = m.newblk[i];
        const NewPlace p = place_of(m, starts, nb, M);
        const int b = (int)nb.bucket;
        m.reqset[nb.setslot] = 0ull;
        m.bucket_cnt[b] = 0;
        if (!fast) {
            m.order[p.rank] = i;
            continue;
        }
        HEntry e;
        e.x = nb.x;
        e.y = nb.y;
        e.z = nb.z;
        e.pad = 0;
        e.ptr = m.heap[hc0 - p.rank];
        int slot;
        if (nb.he && p.among == 0) {
            slot = b;
            e.offset = p.more ? ep0 + p.xbefore : 0;
        } else {
            const int q = p.among - nb.he;        // rank among this bucket's excess blocks
            const int off = ep0 + p.xbefore + q;
            slot = m.NB + off - 1;
            e.offset = p.more ? off + 1 : 0;
            if (q == 0 && !nb.he) {
                // link the tail of the existing chain (CreateBlock's e->offset = offset)
                int t = b;
                for (int guard = 0; m.entries[t].offset > 0 && m.entries[t].offset <= m.NE && guard <= m.NE;
                     ++guard)
                    t = m.NB + m.entries[t].offset - 1;
                m.entries[t].offset = off;
            }
        }
        m.entries[slot] = e;
        m.alloc_list[na0 + p.rank] = slot;
    }
    if (!last_to_finish(&m.bins->ticket, (unsigned)(ctx.gx * ctx.gy))) return;
    if (M > 0)
        for (int i = threadIdx.x; i < kAllocBins; i += blockDim.x) {
            m.bins->cnt[i] = 0;
            m.bins->head[i] = -1;
        }
    if (threadIdx.x != 0) return;
    const int excess = M > 0 ? __ldcg(&c->excess_total) : 0;
    if (M > 0 && M <= hc0 + 1 && ep0 - 1 + excess <= m.NE && !holes0) {
        c->heap_counter = hc0 - M;
        c->entry_ptr = ep0 + excess;
        c->n_alloc = na0 + M;
        c->seq_path = 0;
    } else if (M > 0) {
        int hc = hc0, ep = ep0, holes = holes0, na = na0;
        for (int R = 0; R < M; ++R) {
            const NewBlock nb = m.newblk[__ldcg(&m.order[R])];
            int slot = create_block_seq(m, nb.x, nb.y, nb.z, hc, ep, holes);
            if (slot >= 0 && m.entries[slot].ptr != -1) m.alloc_list[na++] = slot;
        }
        unsigned err = kErrSequentialInsert;
        if (hc < -1) err |= kErrHeapExhausted;
        if (ep - 1 > m.NE) err |= kErrExcessFull;
        atomicOr(&c->err, err);
        c->heap_counter = hc;
        c->entry_ptr = ep;
        c->holes = holes;
        c->n_alloc = na;
        c->seq_path = 1;
    }
    c->n_new = M;
    c->n_req = 0;
    c->n_visible = 0;
    c->n_tiles = 0;
}

__global__ void __launch_bounds__(256) k_alloc_insert(MapView m, int zinit) {
    alloc_insert_body(own_ctx(), m, zinit);
}
FB_FUSED_KERNEL(k_alloc_insert, alloc_insert_body, 256)


// ---------------------------------------------------------------- visibility

__device__ __forceinline__ void reset_visible_body(const BlockCtx& ctx, MapCounters* c) {
    c->n_visible = 0;
    c->n_tiles = 0;
}

__global__ void __launch_bounds__(32) k_reset_visible(MapCounters* c) {
    reset_visible_body(own_ctx(), c);
}
FB_FUSED_KERNEL(k_reset_visible, reset_visible_body, 32)

__device__ __forceinline__ void visibility_body(const BlockCtx& ctx, MapView m, int W, int H, Intr k,
                                                const DevPose* __restrict__ posep, const int* __restrict__ skip) {
    if (skip && *skip) return;
    const DevPose P = *posep;
    const int n = m.ctr->n_alloc;
    const int nIter = (n + ctx.gx * blockDim.x - 1) / (ctx.gx * blockDim.x);
    for (int it = 0; it < nIter; ++it) {
        const int i = (it * ctx.gx + ctx.bx) * blockDim.x + threadIdx.x;
        bool vis = false;
        int slot = -1;
        HEntry e;
        if (i < n) {
            slot = m.alloc_list[i];
            e = m.entries[slot];
            vis = block_visible(e.x, e.y, e.z, P, k, W, H, m.g);
        }
        append_visible(m, vis, slot, e);
    }
}

__global__ void __launch_bounds__(256) k_visibility(MapView m, int W, int H, Intr k,
                                  const DevPose* __restrict__ posep, const int* __restrict__ skip) {
    visibility_body(own_ctx(), m, W, H, k, posep, skip);
}
FB_FUSED_KERNEL(k_visibility, visibility_body, 256)

// --------------------------------------------------------------- integration

// Fusion records of caller images (fb_fuse_map_color; the frame path makes
// them in the level-0 map kernel): see fuse_record.  The integration kernels
// use 1 for the normal's w lane, which ComputeNMap sets on every valid normal
// (Pyrdown.cu:93-125); a valid normal with another w lane is flagged.
__global__ void k_fuse_records(MapView m, const float* __restrict__ raw, int rp, const uint8_t* __restrict__ rgb,
                               int cp, const float4* __restrict__ nmap, int np, int W, int H) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= W || y >= H) return;
    const float4 n = nmap[(size_t)y * np + x];
    if (!isnan(n.x) && n.w != 1.0f) atomicOr(&m.ctr->err, kErrNormalW);
    if (m.cvox)
        fuse_record_packed(raw[(size_t)y * rp + x], n, rgb + (size_t)y * cp + 3 * x, m.g.depth_min, m.g.depth_max,
                           (uint4*)m.frec + (size_t)y * W + x);
    else
        fuse_record(raw[(size_t)y * rp + x], n, rgb + (size_t)y * cp + 3 * x, m.g.depth_min, m.g.depth_max,
                    m.frec + (size_t)y * W + x, m.fcol + (size_t)y * W + x);
}

// Two floats in one register pair (Blackwell's packed FP32: one issue slot for
// both lanes of an operation; each lane is rounded as its scalar form).
using f2 = unsigned long long;
__device__ __forceinline__ f2 f2_of(float a, float b) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float f2_lo(f2 v) {
    float a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
    return a;
}
__device__ __forceinline__ float f2_hi(f2 v) {
    float a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
    return b;
}
__device__ __forceinline__ f2 f2_add(f2 a, f2 b) {
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// Per-launch constants of integrate_pair, both lanes equal.  nz holds -0.0f: a
// product is written a b + (-0), which rounds as a b alone, because the
// compiler merges a packed multiply and the add that follows it into one FMA.
struct PairConst {
    f2 nz, m1;
    f2 nfx, nfy, cx, cy;     // -fx, -fy
    f2 nT, rT;               // -trunc_dist, 1 / trunc_dist
};
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b, const PairConst& pc) { return f2_fma(a, b, pc.nz); }

__device__ __forceinline__ PairConst pair_const(const Intr& k, float T, int W) {
    PairConst pc;
    // not a constant the compiler can fold (W > 0 at every launch)
    const float nz = __uint_as_float(0x80000000u | (W < 0 ? 1u : 0u));
    const float rT = __frcp_rn(T);
    pc.nz = f2_of(nz, nz);
    pc.m1 = f2_of(-1.0f, -1.0f);
    pc.nfx = f2_of(-k.fx, -k.fx);
    pc.nfy = f2_of(-k.fy, -k.fy);
    pc.cx = f2_of(k.cx, k.cx);
    pc.cy = f2_of(k.cy, k.cy);
    pc.nT = f2_of(-T, -T);
    pc.rT = f2_of(rT, rT);
    return pc;
}

// Fusion::integrateColor (FuseMap.cu:140-191) for the voxels (vx, vy, vz) and
// (vx + 1, vy, vz), every operation rounded as the reference's float
// expression.  rec / col: the frame's fusion records (W wide).  Returns true
// when a voxel changed.
//
// Quotients by one divisor share its reciprocal (fd_rcp's correction step
// without its test for a zero remainder, which only keeps the sign of a zero
// quotient: a projected coordinate adds the centre, a normal's component adds
// a positive term, and a signed distance is never -0).  Some are computed
// negated, so that the packed forms need no negation: -(a b) and (-a) b are
// the same bits.
//
// Bound by issue slots (74 % busy at 20 k blocks, DRAM at 1.2 TB/s): two voxels
// a thread share the packed operations.  20 k blocks at 640x480 111 -> 95 us,
// a live 640x480 frame 37 -> 31, against one scalar voxel after the other.
__device__ __forceinline__ bool integrate_pair(Voxel& v0, Voxel& v1, int vx, int vy, int vz,
                                               const float4* __restrict__ rec, const uint32_t* __restrict__ col,
                                               int W, int H, const Intr& k, const DevPose& P, const MapGeom& g,
                                               const float* __restrict__ div255, const PairConst& pc) {
    const float wx0 = fs(fm((float)vx, g.voxel_size), P.t.x), wx1 = fs(fm((float)(vx + 1), g.voxel_size), P.t.x);
    const float wy = fs(fm((float)vy, g.voxel_size), P.t.y), wz = fs(fm((float)vz, g.voxel_size), P.t.z);
    const f3 p0 = mv(P.Rinv, mk3(wx0, wy, wz)), p1 = mv(P.Rinv, mk3(wx1, wy, wz));
    const f2 px = f2_of(p0.x, p1.x), py = f2_of(p0.y, p1.y), pz = f2_of(p0.z, p1.z);
    // u, v = f p / z + c: -a = (-f) p, q = (-a)(-1/z), q z - a = -(remainder)
    f2 pu, pv;
    {
        const f2 nrz = f2_of(__frcp_rn(-p0.z), __frcp_rn(-p1.z));
        const f2 nax = f2_mul(pc.nfx, px, pc), nay = f2_mul(pc.nfy, py, pc);
        const f2 qx = f2_mul(nax, nrz, pc), qy = f2_mul(nay, nrz, pc);
        pu = f2_add(f2_fma(f2_fma(qx, pz, nax), nrz, qx), pc.cx);
        pv = f2_add(f2_fma(f2_fma(qy, pz, nay), nrz, qy), pc.cy);
    }
    int u0 = __float2int_rz(f2_lo(pu)), u1 = __float2int_rz(f2_hi(pu));   // make_int2(float2)
    int w0 = __float2int_rz(f2_lo(pv)), w1 = __float2int_rz(f2_hi(pv));
    if (p0.z == 0.0f) {   // the IEEE quotients by zero
        u0 = __float2int_rz(fa(fd(fm(k.fx, p0.x), p0.z), k.cx));
        w0 = __float2int_rz(fa(fd(fm(k.fy, p0.y), p0.z), k.cy));
    }
    if (p1.z == 0.0f) {
        u1 = __float2int_rz(fa(fd(fm(k.fx, p1.x), p1.z), k.cx));
        w1 = __float2int_rz(fa(fd(fm(k.fy, p1.y), p1.z), k.cy));
    }
    const bool in0 = (unsigned)u0 < (unsigned)W && (unsigned)w0 < (unsigned)H;
    const bool in1 = (unsigned)u1 < (unsigned)W && (unsigned)w1 < (unsigned)H;
    if (!in0 && !in1) return false;
    const int pix0 = in0 ? w0 * W + u0 : 0, pix1 = in1 ? w1 * W + u1 : 0;
    const float4 r0 = __ldg(rec + pix0), r1 = __ldg(rec + pix1);   // .x: the raw depth, NaN where the pixel is skipped
    const uint32_t c0 = __ldg(col + pix0), c1 = __ldg(col + pix1);
    const float s0 = fs(r0.x, p0.z), s1 = fs(r1.x, p1.z);
    const bool on0 = in0 && s0 >= -g.trunc_dist, on1 = in1 && s1 >= -g.trunc_dist;
    if (!on0 && !on1) return false;
    f2 sd = f2_of(s0, s1);
    {
        const f2 q = f2_mul(sd, pc.rT, pc);
        sd = f2_fma(f2_fma(q, pc.nT, sd), pc.rT, q);
    }
    const float sdf0 = fminf(1.0f, f2_lo(sd)), sdf1 = fminf(1.0f, f2_hi(sd));
    sd = f2_of(sdf0, sdf1);
    // w = nl * normalised(float4(pos, 1)): the dot runs over all four lanes
    // (the normal's w lane is 1, so its term is 1 / nrm)
    const f2 nn = f2_add(f2_add(f2_add(f2_mul(px, px, pc), f2_mul(py, py, pc)), f2_mul(pz, pz, pc)),
                         f2_of(1.0f, 1.0f));
    const float n0 = fsq(f2_lo(nn)), n1 = fsq(f2_hi(nn));
    const float rn0 = __frcp_rn(n0), rn1 = __frcp_rn(n1);
    const f2 nrm = f2_of(n0, n1), nrn = f2_of(-rn0, -rn1);
    // minus each component's term (-q = p (-1/n), p - q n, -(q + r / n))
    auto term = [&](f2 p, float a, float b) {
        const f2 nq = f2_mul(p, nrn, pc);
        return f2_mul(f2_of(a, b), f2_fma(f2_fma(nq, nrm, p), nrn, nq), pc);
    };
    const f2 nsum = f2_add(f2_add(term(px, r0.y, r1.y), term(py, r0.z, r1.z)), term(pz, r0.w, r1.w));
    const f2 w = f2_fma(nsum, pc.m1, f2_of(rn0, rn1));
    const f2 a = f2_mul(w, f2_of(0.2f, 0.2f), pc), oa = f2_fma(a, pc.m1, f2_of(1.0f, 1.0f));
    const f2 W0 = f2_of((float)v0.weight, (float)v1.weight);
    // (float)c / 255 of a byte c: the table holds those 256 IEEE quotients
    auto blend = [&](uint32_t ca, uint32_t cb, uint32_t va, uint32_t vb) {
        return f2_mul(f2_add(f2_mul(a, f2_of(div255[ca], div255[cb]), pc),
                             f2_mul(oa, f2_of(div255[va], div255[vb]), pc)),
                      f2_of(255.f, 255.f), pc);
    };
    const f2 rr = blend(c0 & 255u, c1 & 255u, v0.r, v1.r);
    const f2 gg = blend((c0 >> 8) & 255u, (c1 >> 8) & 255u, v0.g, v1.g);
    const f2 bb = blend(c0 >> 16, c1 >> 16, v0.b, v1.b);
    const f2 num = f2_add(f2_mul(f2_of(v0.sdf, v1.sdf), W0, pc), f2_mul(w, sd, pc)), den = f2_add(W0, w);
    // the first observation, else the running average; make_uchar3(float3):
    // truncate to int, then to the low byte
    auto put = [](Voxel& v, float sdf, uint32_t c, float n, float d, float r, float gr, float b) {
        if (v.weight == 0) {
            v.sdf = sdf;
            v.weight = 1;
            v.r = (unsigned char)(c & 255u);
            v.g = (unsigned char)((c >> 8) & 255u);
            v.b = (unsigned char)(c >> 16);
        } else {
            v.sdf = fd(n, d);
            v.weight = (unsigned char)min(255, (int)v.weight + 1);
            v.r = (unsigned char)__float2int_rz(r);
            v.g = (unsigned char)__float2int_rz(gr);
            v.b = (unsigned char)__float2int_rz(b);
        }
    };
    if (on0) put(v0, sdf0, c0, f2_lo(num), f2_lo(den), f2_lo(rr), f2_lo(gg), f2_lo(bb));
    if (on1) put(v1, sdf1, c1, f2_hi(num), f2_hi(den), f2_hi(rr), f2_hi(gg), f2_hi(bb));
    return true;
}

__device__ __forceinline__ void integrate_body(const BlockCtx& ctx, MapView m, int W, int H, Intr k,
                                               const DevPose* __restrict__ posep, const int* __restrict__ skip,
                                               int clear_grid) {
    if (skip && *skip) return;
    if (clear_grid) grid_clear(m, ctx.bx * blockDim.x + threadIdx.x, ctx.gx * blockDim.x);
    __shared__ float s_div255[256];
    s_div255[threadIdx.x] = fd((float)threadIdx.x, 255.f);   // blockDim.x == 256
    __syncthreads();
    const DevPose P = *posep;
    const PairConst pc = pair_const(k, m.g.trunc_dist, W);
    const int n = min(m.ctr->n_visible, m.NS);
    const int t = threadIdx.x;
    const int lx = (2 * t) & 7, ly = (t >> 2) & 7, lz = t >> 5;
    const float4* __restrict__ rec = m.frec;
    const uint32_t* __restrict__ col = m.fcol;
    // the next block's entry and voxels are loaded while this block's voxels
    // are integrated (the blocks of one CTA are distinct)
    HEntry e_nx;
    uint4 raw_nx;
    if (ctx.bx < n) {
        e_nx = m.vis_blocks[ctx.bx];
        raw_nx = *((const uint4*)(m.voxels + (size_t)e_nx.ptr * 512) + t);
    }
    for (int b = ctx.bx; b < n; b += ctx.gx) {
        const HEntry e = e_nx;
        const int vx = e.x * 8 + lx, vy = e.y * 8 + ly, vz = e.z * 8 + lz;
        uint4* base = (uint4*)(m.voxels + (size_t)e.ptr * 512) + t;
        const uint4 raw2 = raw_nx;
        if (b + ctx.gx < n) {
            e_nx = m.vis_blocks[b + ctx.gx];
            raw_nx = *((const uint4*)(m.voxels + (size_t)e_nx.ptr * 512) + t);
        }
        Voxel v0 = *(const Voxel*)&raw2.x, v1 = *(const Voxel*)&raw2.z;
        if (integrate_pair(v0, v1, vx, vy, vz, rec, col, W, H, k, P, m.g, s_div255, pc)) {
            uint4 o;
            *(Voxel*)&o.x = v0;
            *(Voxel*)&o.z = v1;
            *base = o;
        }
    }
}

__global__ void __launch_bounds__(256) k_integrate(MapView m, int W, int H, Intr k, const DevPose* __restrict__ posep,
                                  const int* __restrict__ skip, int clear_grid) {
    integrate_body(own_ctx(), m, W, H, k, posep, skip, clear_grid);
}
FB_FUSED_KERNEL(k_integrate, integrate_body, 256)

// Precision form of k_integrate: 6-byte voxels (FP16 TSDF and one r, g, b,
// weight word), contracted FP32.  One wave of CTAs of 128 threads; each CTA
// takes every gridDim.x-th visible block.  The block's voxel loads are issued
// before the projections, so they overlap the record gathers.  Thread t owns
// four x-consecutive voxels, so its TSDF (8 B) and words (16 B) are two
// coalesced vector loads and stores; which (y, z) it owns is chosen per frame
// so that a warp's 32 voxels of one gather lie along the viewing direction.
// The per-pixel inputs are one packed 16-byte record (fuse_record_packed):
// the gathers, not the voxel traffic, bound this kernel (L1 wavefronts of
// scattered loads), so one gather per voxel instead of two matters most.
// Camera-space positions come from a per-block origin and the columns of
// Rinv scaled by the voxel size (voxel q of the four at origin + q x-column).
//
// The update is integrateColor's (FuseMap.cu:140-191): project (truncated
// pixel), record depth valid, sdf >= -T, sdf = min(1, sdf / T),
// w = n . normalised(p, 1) over four lanes, first observation or weighted
// running average, weight + 1 capped at 255, colour c0 + 0.2 w (c - c0).
// The colour is blended on floats 1.5 * 2^23 + byte, whose low mantissa bits
// are the byte: one exact subtraction and one fused multiply-add rounded
// toward zero give floor(c0 + 0.2 w (c - c0)) modulo 256 (the reference
// truncates toward zero; the two differ only where the sum is negative and
// wraps).
__device__ __forceinline__ float byte_as_magic(uint32_t word, uint32_t sel) {
    // byte `sel` of `word` into the low byte of 0x4b400000 = 1.5 * 2^23
    return __uint_as_float(__byte_perm(word, 0x4b400000u, sel | 0x7650u));
}

__device__ __forceinline__ void integrate_compact_body(const BlockCtx& ctx, MapView m, int W, int H, Intr k,
                                                       const DevPose* __restrict__ posep,
                                                       const int* __restrict__ skip, int clear_grid) {
    if (skip && *skip) return;
    if (clear_grid) grid_clear(m, ctx.bx * blockDim.x + threadIdx.x, ctx.gx * blockDim.x);
    const DevPose P = *posep;
    const int n = min(m.ctr->n_visible, m.NS);
    const int t = threadIdx.x, l = t & 31, wq = t >> 5;
    // voxels of a warp's gather lie along the world axis closest to the
    // viewing direction (the camera's z axis in world coordinates is row 2 of
    // Rinv), where they project onto few pixels: lane bits 1-4 and the warp
    // index split the block's y and z coordinates accordingly; each thread
    // keeps four x-consecutive voxels (vector loads and stores)
    const float ax = fabsf(P.Rinv.r2.x), ay = fabsf(P.Rinv.r2.y), az = fabsf(P.Rinv.r2.z);
    int ly, lz;
    if (az >= ax && az >= ay) {          // view along z: 8 z x 2 y per warp
        ly = ((l >> 1) & 1) | (wq << 1);
        lz = (l >> 2) & 7;
    } else if (ay >= ax) {               // view along y: 8 y x 2 z per warp
        ly = (l >> 1) & 7;
        lz = ((l >> 4) & 1) | (wq << 1);
    } else {                             // view along x: 4 y x 4 z per warp
        ly = ((l >> 1) & 3) | ((wq & 1) << 2);
        lz = ((l >> 3) & 3) | ((wq >> 1) << 2);
    }
    const int lx = 4 * (l & 1);
    const int idx = lz * 64 + ly * 8 + lx;
    const float vs = m.g.voxel_size, T = m.g.trunc_dist, invT = 1.0f / T;
    // camera = Rinv (world - t): basis columns Rinv e_i * vs and offset -Rinv t
    const f3 bx = mk3(P.Rinv.r0.x * vs, P.Rinv.r1.x * vs, P.Rinv.r2.x * vs);
    const f3 by = mk3(P.Rinv.r0.y * vs, P.Rinv.r1.y * vs, P.Rinv.r2.y * vs);
    const f3 bz = mk3(P.Rinv.r0.z * vs, P.Rinv.r1.z * vs, P.Rinv.r2.z * vs);
    const f3 c0 = mk3(-(P.Rinv.r0.x * P.t.x + P.Rinv.r0.y * P.t.y + P.Rinv.r0.z * P.t.z),
                      -(P.Rinv.r1.x * P.t.x + P.Rinv.r1.y * P.t.y + P.Rinv.r1.z * P.t.z),
                      -(P.Rinv.r2.x * P.t.x + P.Rinv.r2.y * P.t.y + P.Rinv.r2.z * P.t.z));
    const uint4* __restrict__ rec = (const uint4*)m.frec;   // packed records (fuse_record_packed)
    for (int b = ctx.bx; b < n; b += ctx.gx) {
        const HEntry e4 = m.vis_blocks[b];
        const int4 e = make_int4(e4.x, e4.y, e4.z, e4.ptr);
        uint8_t* blk = m.cvox + (size_t)e.w * kCBlockBytes;
        uint2 sd = *(const uint2*)(blk + 2 * idx);
        const uint4 cw = *(const uint4*)(blk + kCRgbw + 4 * idx);
        const float ox = (float)(e.x * 8 + lx), oy = (float)(e.y * 8 + ly), oz = (float)(e.z * 8 + lz);
        f3 p;
        p.x = fmaf(bx.x, ox, fmaf(by.x, oy, fmaf(bz.x, oz, c0.x)));
        p.y = fmaf(bx.y, ox, fmaf(by.y, oy, fmaf(bz.y, oz, c0.y)));
        p.z = fmaf(bx.z, ox, fmaf(by.z, oy, fmaf(bz.z, oz, c0.z)));
        // the four projections, then their record gathers issued together;
        // voxel q sits at p + q bx (recomputed where needed: fewer live
        // registers than keeping the four positions)
        int pix[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const f3 pq = mk3(fmaf((float)q, bx.x, p.x), fmaf((float)q, bx.y, p.y), fmaf((float)q, bx.z, p.z));
            const float rz = __fdividef(1.0f, pq.z);
            const int u = __float2int_rz(fmaf(k.fx * pq.x, rz, k.cx));
            const int v = __float2int_rz(fmaf(k.fy * pq.y, rz, k.cy));
            pix[q] = ((unsigned)u < (unsigned)W && (unsigned)v < (unsigned)H) ? v * W + u : -1;
        }
        uint4 r[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) r[q] = pix[q] >= 0 ? __ldg(rec + pix[q]) : make_uint4(0x7fffffffu, 0u, 0u, 0u);
        const __half2 s01 = *(const __half2*)&sd.x, s23 = *(const __half2*)&sd.y;
        float sdf[4] = {__low2float(s01), __high2float(s01), __low2float(s23), __high2float(s23)};
        uint32_t word[4] = {cw.x, cw.y, cw.z, cw.w};
        bool changed = false;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const f3 pq = mk3(fmaf((float)q, bx.x, p.x), fmaf((float)q, bx.y, p.y), fmaf((float)q, bx.z, p.z));
            const float so = __uint_as_float(r[q].x) - pq.z;
            if (!(so >= -T)) continue;   // NaN depth (skipped pixel or outside the image) fails too
            const float ts = fminf(1.0f, so * invT);
            const float2 nxy = __half22float2(*reinterpret_cast<const __half2*>(&r[q].y));
            const float nz = __half2float(__ushort_as_half((unsigned short)(r[q].z & 0xffffu)));
            const uint32_t cq = (r[q].z >> 16) | (r[q].w << 16);   // r | g << 8 | b << 16
            const float w = fmaf(nxy.x, pq.x, fmaf(nxy.y, pq.y, fmaf(nz, pq.z, 1.0f))) *
                            rsqrtf(fmaf(pq.x, pq.x, fmaf(pq.y, pq.y, fmaf(pq.z, pq.z, 1.0f))));
            const uint32_t W0 = word[q] >> 24;
            if (W0 == 0) {
                sdf[q] = ts;
                word[q] = cq | (1u << 24);
            } else {
                const float Wf = (float)W0, a = 0.2f * w;
                sdf[q] = __fdividef(fmaf(sdf[q], Wf, w * ts), Wf + w);
                const float r0 = byte_as_magic(word[q], 0), g0 = byte_as_magic(word[q], 1),
                            b0 = byte_as_magic(word[q], 2);
                const float rn = __fmaf_rz(a, byte_as_magic(cq, 0) - r0, r0);
                const float gn = __fmaf_rz(a, byte_as_magic(cq, 1) - g0, g0);
                const float bn = __fmaf_rz(a, byte_as_magic(cq, 2) - b0, b0);
                const uint32_t rg = __byte_perm(__float_as_uint(rn), __float_as_uint(gn), 0x0040u);
                const uint32_t bw = __byte_perm(__float_as_uint(bn), (W0 < 255u ? W0 + 1u : 255u), 0x0040u);
                word[q] = __byte_perm(rg, bw, 0x5410u);
            }
            changed = true;
        }
        if (changed) {
            const __half2 n01 = __floats2half2_rn(sdf[0], sdf[1]), n23 = __floats2half2_rn(sdf[2], sdf[3]);
            sd.x = *(const uint32_t*)&n01;
            sd.y = *(const uint32_t*)&n23;
            *(uint2*)(blk + 2 * idx) = sd;
            *(uint4*)(blk + kCRgbw + 4 * idx) = make_uint4(word[0], word[1], word[2], word[3]);
        }
    }
}

__global__ void __launch_bounds__(128, 7) k_integrate_compact(MapView m, int W, int H, Intr k,
                                  const DevPose* __restrict__ posep, const int* __restrict__ skip,
                                  int clear_grid) {
    integrate_compact_body(own_ctx(), m, W, H, k, posep, skip, clear_grid);
}
FB_FUSED_KERNEL(k_integrate_compact, integrate_compact_body, 128, 7)

// ------------------------------------------------- the reference's layouts

// The reference's HashEntry (Mapping/DeviceMap.h:17-59, __align__(16): 32
// bytes): block position, voxel index of the block (block * 512) or -1, and
// the chain offset.
struct RefHashEntry {
    int x, y, z, ptr, offset, pad[3];
};
static_assert(sizeof(RefHashEntry) == 32, "the reference's HashEntry");

__device__ __forceinline__ RefHashEntry to_ref_entry(const HEntry& e) {
    RefHashEntry r;
    r.x = e.x;
    r.y = e.y;
    r.z = e.z;
    r.ptr = e.ptr >= 0 ? e.ptr * 512 : -1;
    r.offset = e.offset;
    r.pad[0] = r.pad[1] = r.pad[2] = 0;
    return r;
}

// n entries (from a table or the visible list) in the reference's layout.
__global__ void k_export_ref_entries(const HEntry* __restrict__ src, const int* __restrict__ count, int n,
                                     RefHashEntry* __restrict__ dst) {
    const int lim = count ? min(*count, n) : n;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < lim; i += gridDim.x * blockDim.x)
        dst[i] = to_ref_entry(src[i]);
}

// Precision-form voxels in the reference's 8-byte Voxel layout (FP16 TSDF
// widened to float).
__global__ void k_export_ref_voxels(MapView m, Voxel* __restrict__ dst) {
    const size_t n = (size_t)m.NS * 512;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const uint8_t* blk = m.cvox + (i / 512) * kCBlockBytes;
        const int v = (int)(i % 512);
        Voxel o;
        o.sdf = __half2float(reinterpret_cast<const __half*>(blk)[v]);
        const uint32_t w = *reinterpret_cast<const uint32_t*>(blk + kCRgbw + 4 * v);
        o.weight = (uint8_t)(w >> 24);
        o.r = (uint8_t)w;
        o.g = (uint8_t)(w >> 8);
        o.b = (uint8_t)(w >> 16);
        dst[i] = o;
    }
}

__global__ void k_export_ref_counters(const MapCounters* __restrict__ c, int* heap_counter, int* entry_ptr) {
    if (heap_counter) *heap_counter = c->heap_counter;
    if (entry_ptr) *entry_ptr = c->entry_ptr;
}

// ---------------------------------------------------------------------- reset

// ResetHashKernel / ResetSdfBlockKernel (FuseMap.cu:321-350) on all of the
// table (the reference leaves pos and offset of released entries in place).
__global__ void k_map_reset(MapView m) {
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    const size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t ne = (size_t)m.NB + m.NE;
    for (size_t i = tid; i < ne; i += stride) {
        HEntry e;
        e.x = e.y = e.z = e.pad = 0;
        e.ptr = -1;
        e.offset = 0;
        m.entries[i] = e;
    }
    for (size_t i = tid; i < (size_t)m.NS; i += stride) m.heap[i] = m.NS - (int)i - 1;
    if (m.cvox) {
        // precision form: FP16 NaN TSDF, weight 0, colour 0 (64 + 128 uint4 per block)
        const uint4 nan8 = make_uint4(0x7e007e00u, 0x7e007e00u, 0x7e007e00u, 0x7e007e00u);
        const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
        uint4* vv = (uint4*)m.cvox;
        for (size_t i = tid; i < (size_t)m.NS * (kCBlockBytes / 16); i += stride)
            vv[i] = (i % (kCBlockBytes / 16)) < 64 ? nan8 : zero;
    } else {
        const uint4 released = make_uint4(0x7fffffffu, 0u, 0x7fffffffu, 0u);  // {NaN, w 0, rgb 0} x 2
        uint4* vv = (uint4*)m.voxels;
        for (size_t i = tid; i < (size_t)m.NS * 256; i += stride) vv[i] = released;
    }
    for (size_t i = tid; i < (size_t)m.NB; i += stride) m.bucket_cnt[i] = 0;
    for (size_t i = tid; i < (size_t)m.reqcap; i += stride) m.reqset[i] = 0ull;
    for (size_t i = tid; i < (size_t)kAllocBins; i += stride) {
        m.bins->cnt[i] = 0;
        m.bins->head[i] = -1;
    }
    if (tid == 0) {
        m.bins->ticket = 0;
        MapCounters* c = m.ctr;
        c->heap_counter = m.NS - 1;
        c->entry_ptr = 1;
        c->holes = 0;
        c->n_alloc = 0;
        c->n_req = 0;
        c->n_new = 0;
        c->n_visible = 0;
        c->n_tiles = 0;
        c->excess_total = 0;
        c->err = 0;
        c->seq_path = 0;
        c->ray_next = 0;
    }
}

// ------------------------------------------------------------------ launchers

static int sm_count() {
    static int n = 0;
    if (!n) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        if (n <= 0) n = 148;
    }
    return n;
}

int launch_map_reset(const MapView& m, cudaStream_t s) { k_map_reset<<<sm_count() * 8, 256, 0, s>>>(m);
    return 1;
}

int launch_allocate(const MapView& m, const float* raw, int rp, int W, int H, const Intr& k, const DevPose* pose,
                     const int* skip, cudaStream_t s, bool zinit) {
    dim3 b(32, 8), g((W + 31) / 32, (H + 7) / 8);
    fb_launch(k_alloc_requests, (const void*)k_alloc_requests_fused, g, b, 0, s, m, raw, rp, W, H, k, pose, skip);
    fb_launch(k_alloc_insert, (const void*)k_alloc_insert_fused, sm_count() * 2, 256, 0, s, m, zinit ? 1 : 0);
    return 2;
}

int launch_visibility(const MapView& m, int W, int H, const Intr& k, const DevPose* pose, const int* skip,
                       cudaStream_t s, bool after_allocate) {
    // the allocation's last kernel (k_alloc_insert) zeroes the same counters
    if (!after_allocate) fb_launch(k_reset_visible, (const void*)k_reset_visible_fused, 1, 1, 0, s, m.ctr);
    fb_launch(k_visibility, (const void*)k_visibility_fused, sm_count() * 4, 256, 0, s, m, W, H, k, pose, skip);
    return after_allocate ? 1 : 2;
}

int launch_export_visible(const MapView& m, void* dst, int capacity, cudaStream_t s) {
    k_export_ref_entries<<<sm_count() * 2, 256, 0, s>>>(m.vis_blocks, &m.ctr->n_visible, min(capacity, m.NS),
                                                          (RefHashEntry*)dst);
    return 1;
}

int launch_export_reference(const MapView& m, void* entries, void* voxels, int* heap_counter, int* entry_ptr,
                            cudaStream_t s) {
    k_export_ref_entries<<<sm_count() * 8, 256, 0, s>>>(m.entries, nullptr, m.NB + m.NE, (RefHashEntry*)entries);
    if (m.cvox) k_export_ref_voxels<<<sm_count() * 8, 256, 0, s>>>(m, (Voxel*)voxels);
    k_export_ref_counters<<<1, 1, 0, s>>>(m.ctr, heap_counter, entry_ptr);
    return m.cvox ? 3 : 2;
}

int launch_fuse_records(const MapView& m, const float* raw, int rp, const uint8_t* rgb, int cp, const float4* nmap,
                        int np, int W, int H, cudaStream_t s) {
    dim3 b(32, 8), g((W + 31) / 32, (H + 7) / 8);
    k_fuse_records<<<g, b, 0, s>>>(m, raw, rp, rgb, cp, nmap, np, W, H);
    return 1;
}

int launch_integrate(const MapView& m, int W, int H, const Intr& k, const DevPose* pose, const int* skip,
                     cudaStream_t s, int ctas_per_sm, bool clear_grid) {
    const int clear = clear_grid ? 1 : 0;
    const int ctas = sm_count() * (ctas_per_sm ? ctas_per_sm : m.cvox ? 7 : 8);
    if (m.cvox)
        fb_launch(k_integrate_compact, (const void*)k_integrate_compact_fused, ctas, 128, 0, s, m, W, H, k, pose,
                  skip, clear);
    else
        fb_launch(k_integrate, (const void*)k_integrate_fused, ctas, 256, 0, s, m, W, H, k, pose, skip, clear);
    return 1;
}

}  // namespace fb
