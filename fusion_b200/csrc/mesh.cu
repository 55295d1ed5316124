// Marching-cubes mesh extraction of the map (MeshScene, Mapping/MeshScene.cu:
// 20-355, called by Mapping::CreateModel, Mapping.cc:131-140) and the ASCII
// PLY writer of System::WriteMeshToDisk (Core/System.cc:140-193).
//
// Per voxel of every allocated block, as the reference: the cube of the voxel
// and its +x/+y/+z neighbours (any corner missing, NaN or exactly 1.0 -> no
// cube), central-difference gradients at the corners from the 24 voxels
// around the cube (any NaN -> no cube), the case index from sdf < 0, and on
// every cut edge the reference's vertex: interpolation parameter, position
// (voxel + offset) * voxel size, normal = normalised gradient interpolated
// along the edge, colour by the reference's uchar3 arithmetic.
//
// The case table is this library's own construction (build_case): on each
// cube face the cut edges are paired -- a face whose two negative corners sit
// on a diagonal keeps them apart -- and oriented so that the negative side
// lies to the left seen from outside the cube; the pairs close into loops
// across the faces and each loop is triangulated without chords lying in a
// cube face.  Every cut edge
// carries a vertex and two cubes sharing a face pair that face's edges the
// same way, so the mesh is closed wherever the field is defined.  The
// reference's vertices are reproduced exactly; the triangulation of a cube's
// polygon may differ from the reference's table (and the reference's
// classic table leaves holes on some ambiguous faces).  Triangles wind so
// that their right-hand normal points to the negative side.
//
// GPU layout: CTAs of 288 threads walk the allocated blocks.  A CTA stages the
// 11^3 voxel region the block's cubes and gradients read (local coordinates
// -1 .. 9) in shared memory, instead of the reference's 32 hash lookups per
// voxel; the 27 blocks it comes from are looked up by a warp of their own while
// the block before is worked on.  Which voxels hold surface is found a row of
// eight at a time, from a word of bits per row of the region.  Two passes make the output deterministic: triangle
// counts per block, an exclusive scan, then every block writes its triangles
// at its offset in voxel order.  In the second pass the block's triangles are
// listed first and then every thread makes a vertex (few voxels of a block
// hold surface), and the vertices leave through shared memory in whole words.
#include <cstdio>
#include <cstring>
#include <mutex>
#include <vector>

#include <cuda_fp16.h>

#include "../../include/fusion_b200.h"
#include "fb_internal.h"

namespace fb {

// ---------------------------------------------------------------- tables

// Corners (MeshScene.cu:105-140) and the twelve edges of buildVertexList
// (MeshScene.cu:185-256), as corner pairs in the reference's direction.
__host__ __device__ constexpr int corner_dx(int i) { return i == 1 || i == 2 || i == 5 || i == 6; }
__host__ __device__ constexpr int corner_dy(int i) { return i == 2 || i == 3 || i == 6 || i == 7; }
__host__ __device__ constexpr int corner_dz(int i) { return i >= 4; }
__host__ __device__ constexpr int edge_a(int e) { return e < 8 ? e : e - 8; }
__host__ __device__ constexpr int edge_b(int e) { return e < 8 ? ((e & 3) == 3 ? e - 3 : e + 1) : e - 4; }

static int edge_of(int a, int b) {
    for (int e = 0; e < 12; ++e)
        if ((edge_a(e) == a && edge_b(e) == b) || (edge_a(e) == b && edge_b(e) == a)) return e;
    return -1;
}

// Edges e and f lie on a common face of the cube.
static bool share_face(int e, int f) {
    const int a = edge_a(e), b = edge_b(e), c = edge_a(f), d = edge_b(f);
    const int ca[3] = {corner_dx(a), corner_dy(a), corner_dz(a)}, cb[3] = {corner_dx(b), corner_dy(b), corner_dz(b)};
    const int cc[3] = {corner_dx(c), corner_dy(c), corner_dz(c)}, cd[3] = {corner_dx(d), corner_dy(d), corner_dz(d)};
    for (int k = 0; k < 3; ++k)
        if (ca[k] == cb[k] && cc[k] == cd[k] && ca[k] == cc[k]) return true;
    return false;
}

// Triangulates the loop's sub-polygon loop[i .. j] (a polygon side or
// diagonal joins i and j) with diagonals that never join two vertices on
// one cube face: such a chord would lie in the face and, when the
// neighbouring cube draws the same chord, give an edge with four triangles.
// Triangles keep the loop's orientation.  Returns false if impossible.
static bool triangulate(const int* loop, int m, int i, int j, int8_t* tri, int* n) {
    if (j - i < 2) return true;
    auto allowed = [&](int p, int q) { return q == p + 1 || (p == 0 && q == m - 1) || !share_face(loop[p], loop[q]); };
    for (int k = i + 1; k < j; ++k) {
        if (!allowed(i, k) || !allowed(k, j)) continue;
        const int saved = *n;
        if (*n == 5) return false;
        tri[3 * *n + 0] = (int8_t)loop[i];
        tri[3 * *n + 1] = (int8_t)loop[k];
        tri[3 * *n + 2] = (int8_t)loop[j];
        ++*n;
        if (triangulate(loop, m, i, k, tri, n) && triangulate(loop, m, k, j, tri, n)) return true;
        *n = saved;
    }
    return false;
}

// The triangles of cube case `ci` (bit i set: corner i has sdf < 0) as edge
// triples; returns their number (at most 5) or -1 if the construction fails
// (it does not for any case; the tests check all 256).
int build_case(int ci, int8_t tri[16]) {
    // faces as corner quadruples, counter-clockwise seen from outside the cube
    int faces[6][4] = {{0, 3, 2, 1}, {4, 5, 6, 7}, {0, 1, 5, 4}, {3, 7, 6, 2}, {0, 4, 7, 3}, {1, 2, 6, 5}};
    const int outward[6][3] = {{0, 0, -1}, {0, 0, 1}, {0, -1, 0}, {0, 1, 0}, {-1, 0, 0}, {1, 0, 0}};
    for (int f = 0; f < 6; ++f) {   // orientation check of the list above
        const int* q = faces[f];
        int u[3], v[3];
        for (int k = 0; k < 3; ++k) {
            const int c0[3] = {corner_dx(q[0]), corner_dy(q[0]), corner_dz(q[0])};
            const int c1[3] = {corner_dx(q[1]), corner_dy(q[1]), corner_dz(q[1])};
            const int c2[3] = {corner_dx(q[2]), corner_dy(q[2]), corner_dz(q[2])};
            u[k] = c1[k] - c0[k];
            v[k] = c2[k] - c1[k];
        }
        const int c[3] = {u[1] * v[2] - u[2] * v[1], u[2] * v[0] - u[0] * v[2], u[0] * v[1] - u[1] * v[0]};
        if (c[0] * outward[f][0] + c[1] * outward[f][1] + c[2] * outward[f][2] <= 0) return -1;
    }
    auto neg = [ci](int corner) { return (ci >> corner) & 1; };
    // next[e]: the cut edge that follows e along the polygon boundary
    int next[12];
    for (int e = 0; e < 12; ++e) next[e] = -1;
    for (int f = 0; f < 6; ++f) {
        const int* q = faces[f];
        int n_neg = 0;
        for (int k = 0; k < 4; ++k) n_neg += neg(q[k]);
        if (n_neg == 0 || n_neg == 4) continue;
        const bool diagonal = n_neg == 2 && neg(q[0]) == neg(q[2]);
        for (int k = 0; k < 4; ++k) {
            const int a = q[k], b = q[(k + 1) & 3];
            if (!(neg(a) && !neg(b))) continue;
            // leaving the negative region at edge (a, b): walk on around the
            // face (counter-clockwise) to where it is entered again, or, on a
            // diagonal face, close off corner a alone
            int en;
            if (diagonal) {
                en = edge_of(q[(k + 3) & 3], a);
            } else {
                int j = (k + 1) & 3;
                while (!(!neg(q[j]) && neg(q[(j + 1) & 3]))) j = (j + 1) & 3;
                en = edge_of(q[j], q[(j + 1) & 3]);
            }
            const int ex = edge_of(a, b);
            if (next[ex] != -1) return -1;
            next[ex] = en;
        }
    }
    int n = 0;
    bool used[12] = {};
    for (int s = 0; s < 12; ++s) {
        if (next[s] < 0 || used[s]) continue;
        int loop[12], m = 0;
        int e = s;
        while (!used[e]) {
            used[e] = true;
            loop[m++] = e;
            e = next[e];
            if (e < 0) return -1;
        }
        if (e != s || m < 3) return -1;
        if (!triangulate(loop, m, 0, m - 1, tri, &n)) return -1;
    }
    for (int e = 0; e < 12; ++e)   // every cut edge is on a loop
        if (neg(edge_a(e)) != neg(edge_b(e)) && !used[e]) return -1;
    for (int i = 3 * n; i < 16; ++i) tri[i] = -1;
    return n;
}

// (global memory, copied to shared memory by each CTA: constant memory serves
// one address at a time, and every lane reads its own case)
__device__ __align__(16) int8_t c_tri[256][16];
__device__ __align__(16) uint8_t c_ntri[256];

static int build_tables(int8_t tri[256][16], int ntri[256]) {
    for (int ci = 0; ci < 256; ++ci) {
        ntri[ci] = build_case(ci, tri[ci]);
        if (ntri[ci] < 0) return FB_EINVAL;
    }
    return FB_OK;
}

// Uploads the tables to the current device once.
static int ensure_tables() {
    static std::mutex lock;
    static bool done[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return FB_ECUDA;
    std::lock_guard<std::mutex> guard(lock);
    if (done[dev]) return FB_OK;
    int8_t tri[256][16];
    int ntri[256];
    uint8_t n8[256];
    if (build_tables(tri, ntri) != FB_OK) return FB_EINVAL;
    for (int i = 0; i < 256; ++i) n8[i] = (uint8_t)ntri[i];
    if (cudaMemcpyToSymbol(c_tri, tri, sizeof tri) != cudaSuccess) return FB_ECUDA;
    if (cudaMemcpyToSymbol(c_ntri, n8, sizeof n8) != cudaSuccess) return FB_ECUDA;
    done[dev] = true;
    return FB_OK;
}

// ---------------------------------------------------------------- kernels

constexpr int kMeshWork = 256;                     // threads on voxels and vertices ...
constexpr int kMeshThreads = kMeshWork + 32;       // ... and the warp that looks blocks up
constexpr int kMeshCtas = 7;                       // resident per SM (five: 97 us for the triangles, seven: 95)
constexpr int kHalo = 11;                          // local coordinates -1 .. 9
constexpr int kRows = kHalo * kHalo;
constexpr int kRegion = kHalo * kRows;             // 1331
constexpr int kEach = (kRegion + kMeshWork - 1) / kMeshWork;

struct MeshSmem {
    int ptr[2][27];              // blocks around one, (dx + 1) + 3 (dy + 1) + 9 (dz + 1): this block's, the next one's
    int3 pos[2];                 // their block coordinates
    float sdf[kRegion];          // NaN where no block (Voxel(), DeviceMap.h:63-65)
    uint32_t row[kRows];         // the rows' voxels as bits (see row_bits)
    alignas(16) uint8_t ntri[256];
};
// The second pass's additions.
struct EmitSmem {
    uint32_t rgb[kRegion];
    uint16_t tri[512 * 5];       // the block's triangles in order: voxel | triangle of the voxel << 9
    uint8_t cubes[512];          // the voxels' cases
    float v[kMeshWork * 3], n[kMeshWork * 3];
    uint8_t c[kMeshWork * 3];
    alignas(16) int8_t table[256][16];
};

// Barrier of the voxel threads alone (the look-up warp does not take part).
__device__ __forceinline__ void work_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(kMeshWork) : "memory"); }

// FindEntry (DeviceMap.cu:122-135): block index of block (x, y, z), or -1.
__device__ int find_block(const MapView& m, int x, int y, int z) {
    const int b = (int)bucket_of_m(x, y, z, (uint32_t)m.NB, m.nb_mask);
    HEntry e = m.entries[b];
    if (e.ptr != -1 && e.x == x && e.y == y && e.z == z) return e.ptr;
    for (int guard = 0; e.offset > 0 && e.offset <= m.NE && guard <= m.NE; ++guard) {
        e = m.entries[m.NB + e.offset - 1];
        if (e.x == x && e.y == y && e.z == z && e.ptr != -1) return e.ptr;
    }
    return -1;
}

// One lane (< 27) of the look-up warp: a block around allocated block `blk`.
__device__ __forceinline__ void look_up(const MapView& m, int blk, int lane, MeshSmem& s, int buf) {
    if (lane >= 27) return;
    const HEntry self = m.entries[m.alloc_list[blk]];
    const int dx = lane % 3 - 1, dy = (lane / 3) % 3 - 1, dz = lane / 9 - 1;
    // the block itself is looked up too: a map with duplicate entries
    // for one block (the reference's racy allocator makes them) reads the
    // first one, as FindVoxel does
    s.ptr[buf][lane] = find_block(m, self.x + dx, self.y + dy, self.z + dz);
    if (lane == 0) s.pos[buf] = make_int3(self.x, self.y, self.z);
}

// Where a thread's region voxels lie, the same for every block: slot in s.ptr
// << 9 | voxel, or -1 beyond the region.
struct Region {
    int at[kEach];
};
__device__ __forceinline__ Region region_of(int t) {
    Region g;
#pragma unroll
    for (int q = 0; q < kEach; ++q) {
        const int r = t + q * kMeshWork;
        const int lx = r % kHalo - 1, ly = (r / kHalo) % kHalo - 1, lz = r / kRows - 1;
        const int ox = lx < 0 ? -1 : (lx > 7 ? 1 : 0);
        const int oy = ly < 0 ? -1 : (ly > 7 ? 1 : 0);
        const int oz = lz < 0 ? -1 : (lz > 7 ? 1 : 0);
        g.at[q] = r < kRegion ? ((ox + 1) + 3 * (oy + 1) + 9 * (oz + 1)) << 9 |
                                    ((lz - 8 * oz) * 64 + (ly - 8 * oy) * 8 + (lx - 8 * ox))
                              : -1;
    }
    return g;
}

// A row's eleven voxels (local x = -1 .. 9): bits 0-10 the TSDF is not NaN,
// 11-19 (local 0 .. 8) nor exactly 1, 20-28 (local 0 .. 8) it is negative.
__device__ __forceinline__ uint32_t row_bits(const float* sdf) {
    uint32_t b = 0;
#pragma unroll
    for (int u = 0; u < kHalo; ++u) {
        const float v = sdf[u];
        if (!isnan(v)) b |= 1u << u;
        if (u >= 1 && u <= 9) {
            if (!isnan(v) && v != 1.0f) b |= 1u << (10 + u);
            if (v < 0) b |= 1u << (19 + u);
        }
    }
    return b;
}

// The region of the block whose neighbours are in s.ptr[buf] and its rows'
// bits (voxel threads): a thread's voxels are loaded together, then stored.
template <bool kColour>
__device__ __forceinline__ void stage_block(const MapView& m, const Region& g, MeshSmem& s, uint32_t* rgb, int buf) {
    float sdf[kEach];
    uint32_t col[kEach];
#pragma unroll
    for (int q = 0; q < kEach; ++q) {
        sdf[q] = qnan();
        col[q] = 0;
        if (g.at[q] < 0) continue;
        const int p = s.ptr[buf][g.at[q] >> 9], idx = g.at[q] & 511;
        if (p < 0) continue;
        if (m.cvox) {
            const uint8_t* blk = m.cvox + (size_t)p * kCBlockBytes;
            sdf[q] = __half2float(reinterpret_cast<const __half*>(blk)[idx]);
            if (kColour) col[q] = *reinterpret_cast<const uint32_t*>(blk + kCRgbw + 4 * idx) & 0xffffffu;
        } else if (kColour) {
            const uint2 vx = *reinterpret_cast<const uint2*>(m.voxels + (size_t)p * 512 + idx);
            sdf[q] = __uint_as_float(vx.x);
            col[q] = vx.y >> 8;   // weight in the low byte, then r, g, b
        } else {
            sdf[q] = m.voxels[(size_t)p * 512 + idx].sdf;
        }
    }
#pragma unroll
    for (int q = 0; q < kEach; ++q) {
        if (g.at[q] < 0) continue;
        s.sdf[threadIdx.x + q * kMeshWork] = sdf[q];
        if (kColour) rgb[threadIdx.x + q * kMeshWork] = col[q];
    }
    work_barrier();
    if (threadIdx.x < kRows) s.row[threadIdx.x] = row_bits(s.sdf + kHalo * threadIdx.x);
    work_barrier();
}

// Region index of local voxel (x, y, z), each in -1 .. 9.
__device__ __forceinline__ int rix(int x, int y, int z) { return (x + 1) + kHalo * (y + 1) + kRows * (z + 1); }

// The cubes of a block's row (y, z) that hold surface, a bit each, and the
// row's four corner rows: readVertexAndColor + readNormal's NaN tests
// (MeshScene.cu:43-183) for the row's eight voxels together.
struct CubeRow {
    uint32_t mask, r00, r10, r01, r11;   // rdydz: rows (y + dy, z + dz)
};
__device__ __forceinline__ CubeRow cube_row(const MeshSmem& s, int y, int z) {
    const uint32_t* r = s.row + (y + 1) + kHalo * (z + 1);
    CubeRow c;
    c.r00 = r[0];
    c.r10 = r[1];
    c.r01 = r[kHalo];
    c.r11 = r[kHalo + 1];
    const uint32_t all = c.r00 & c.r10 & c.r01 & c.r11, any = c.r00 | c.r10 | c.r01 | c.r11;
    // the 24 gradient neighbours outside the cube: x - 1 and x + 2 of the four
    // rows, and x and x + 1 of the rows beyond them in y and in z
    const uint32_t out = r[-1] & r[2] & r[kHalo - 1] & r[kHalo + 2] & r[-kHalo] & r[-kHalo + 1] & r[2 * kHalo] &
                         r[2 * kHalo + 1];
    const uint32_t ok = all >> 11, nn = out >> 1, na = all >> 20, no = any >> 20;
    c.mask = ok & (ok >> 1) & all & (all >> 3) & nn & (nn >> 1) & (no | (no >> 1)) & ~(na & (na >> 1)) & 0xffu;
    return c;
}
// The case index of the row's cube x (bit i: corner i is negative).
__device__ __forceinline__ int cube_case(const CubeRow& c, int x) {
    const uint32_t a = c.r00 >> (20 + x), b = c.r10 >> (20 + x), d = c.r01 >> (20 + x), e = c.r11 >> (20 + x);
    return (a & 3) | (b & 2) << 1 | (b & 1) << 3 | (d & 3) << 4 | (e & 2) << 5 | (e & 1) << 7;
}

// interp (MeshScene.cu:142-150).  The reference compares in double; for a
// float f, (double)f < 1e-6 exactly when f <= 1e-6f (the float below 1e-6).
__device__ __forceinline__ float interp(float v1, float v2) {
    if (fabsf(v1) <= 1e-6f) return 0.f;
    if (fabsf(v2) <= 1e-6f) return 1.f;
    if (fabsf(fs(v1, v2)) <= 1e-6f) return 0.f;
    return fd(fs(0.f, v1), fs(v2, v1));
}

// Central-difference gradient at corner i (readNormal, MeshScene.cu:43-103).
__device__ __forceinline__ f3 corner_gradient(const MeshSmem& s, int x, int y, int z, int i) {
    const int cx = x + corner_dx(i), cy = y + corner_dy(i), cz = z + corner_dz(i);
    return mk3(fs(s.sdf[rix(cx + 1, cy, cz)], s.sdf[rix(cx - 1, cy, cz)]),
               fs(s.sdf[rix(cx, cy + 1, cz)], s.sdf[rix(cx, cy - 1, cz)]),
               fs(s.sdf[rix(cx, cy, cz + 1)], s.sdf[rix(cx, cy, cz - 1)]));
}

// One vertex of edge e (buildVertexList, MeshScene.cu:185-256, and the
// scaling / normalisation of MarchingCube, MeshScene.cu:284-292).
// normal: n_a + val (n_b - n_a) as one fused multiply-add per component,
// then n / sqrt(n . n) with n . n = fma(z, z, fma(y, y, x x)).
// colour: c_a + (int)val * (c_b - c_a) in bytes (operator*(int, uchar3)).
__device__ __forceinline__ void edge_vertex(const MeshSmem& s, const uint32_t* rgb, int x, int y, int z, int3 g, int e,
                                            float vs, float* V, float* N, uint8_t* C) {
    const int a = edge_a(e), b = edge_b(e);
    const float val = interp(s.sdf[rix(x + corner_dx(a), y + corner_dy(a), z + corner_dz(a))],
                             s.sdf[rix(x + corner_dx(b), y + corner_dy(b), z + corner_dz(b))]);
    // position: the corner a coordinates, the moving axis a's coordinate +/- val
    const int ax = corner_dx(a), ay = corner_dy(a), az = corner_dz(a);
    const int dx = corner_dx(b) - ax, dy = corner_dy(b) - ay, dz = corner_dz(b) - az;
    const float mv = (dx + dy + dz) > 0 ? val : fs(1.f, val);
    const float px = dx ? mv : (float)ax, py = dy ? mv : (float)ay, pz = dz ? mv : (float)az;
    V[0] = fm(fa((float)(g.x + x), px), vs);
    V[1] = fm(fa((float)(g.y + y), py), vs);
    V[2] = fm(fa((float)(g.z + z), pz), vs);
    const f3 na = corner_gradient(s, x, y, z, a), nb = corner_gradient(s, x, y, z, b);
    const f3 n = mk3(__fmaf_rn(val, fs(nb.x, na.x), na.x), __fmaf_rn(val, fs(nb.y, na.y), na.y),
                     __fmaf_rn(val, fs(nb.z, na.z), na.z));
    const float len = fsq(__fmaf_rn(n.z, n.z, __fmaf_rn(n.y, n.y, fm(n.x, n.x))));
    N[0] = fd(n.x, len);
    N[1] = fd(n.y, len);
    N[2] = fd(n.z, len);
    const uint32_t ca = rgb[rix(x + ax, y + ay, z + az)];
    const uint32_t cb = rgb[rix(x + corner_dx(b), y + corner_dy(b), z + corner_dz(b))];
    const int k = (int)val;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const uint8_t ua = (uint8_t)(ca >> (8 * c)), ub = (uint8_t)(cb >> (8 * c));
        C[c] = (uint8_t)(ua + (uint8_t)((uint8_t)(ub - ua) * k));
    }
}

// The walk both passes share: CTA c takes blocks c, c + grid, ...; body(blk,
// buf) runs in the voxel threads, while the look-up warp prepares the next.
template <class Body>
__device__ __forceinline__ void walk_blocks(const MapView& m, int n, MeshSmem& s, Body body) {
    const bool worker = threadIdx.x < kMeshWork;
    int buf = 0;
    if (!worker && (int)blockIdx.x < n) look_up(m, blockIdx.x, threadIdx.x - kMeshWork, s, 0);
    __syncthreads();
    for (int blk = blockIdx.x; blk < n; blk += gridDim.x, buf ^= 1) {
        if (worker)
            body(blk, buf);
        else if (blk + (int)gridDim.x < n)
            look_up(m, blk + gridDim.x, threadIdx.x - kMeshWork, s, buf ^ 1);
        __syncthreads();
    }
}

// Triangle counts of the allocated blocks.  The cubes are found a row of eight
// at a time from bits (cube_row): two warps then walk the few that hold
// surface.  10 800 blocks: 29 us; classifying every voxel from its 32 values
// took 45, and one CTA of 512 threads per block, each beginning with its own
// chain of list, entry and buckets, 83.
__global__ void __launch_bounds__(kMeshThreads, kMeshCtas) k_mesh_count(MapView m, uint2* counts) {
    __shared__ MeshSmem s;
    const int n = min(m.ctr->n_alloc, m.NS), t = threadIdx.x;
    const Region g = region_of(t);
    if (t < 64) reinterpret_cast<uint32_t*>(s.ntri)[t] = reinterpret_cast<const uint32_t*>(c_ntri)[t];
    walk_blocks(m, n, s, [&](int blk, int buf) {
        stage_block<false>(m, g, s, nullptr, buf);
        if (t >= 64) return;
        const CubeRow c = cube_row(s, t & 7, t >> 3);
        int nt = 0;
        for (uint32_t k = c.mask; k; k &= k - 1) nt += s.ntri[cube_case(c, __ffs(k) - 1)];
        __syncwarp();
        nt = __reduce_add_sync(0xffffffffu, nt);
        if ((t & 31) == 0) reinterpret_cast<uint32_t*>(counts)[2 * blk + (t >> 5)] = (uint32_t)nt;
    });
}

// Exclusive scan of the n counts (two halves each) into offsets[0 .. n] (offsets[n] = *total): one
// CTA, each thread a run of consecutive counts.
__global__ void __launch_bounds__(1024) k_mesh_scan(const MapView m, const uint2* counts,
                                                    unsigned long long* offsets, unsigned long long* total) {
    __shared__ unsigned long long warp_sum[32];
    const int n = min(m.ctr->n_alloc, m.NS);
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const int per = (n + 1023) / 1024, i0 = min(n, t * per), i1 = min(n, i0 + per);
    unsigned long long sum = 0;
#pragma unroll 8
    for (int i = i0; i < i1; ++i) sum += counts[i].x + counts[i].y;
    unsigned long long incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) warp_sum[w] = incl;
    __syncthreads();
    unsigned long long run = incl - sum;
    for (int q = 0; q < w; ++q) run += warp_sum[q];
#pragma unroll 8
    for (int i = i0; i < i1; ++i) {
        offsets[i] = run;
        run += counts[i].x + counts[i].y;
    }
    if (t == 1023) offsets[n] = *total = run;
}

// The voxel threads' `bytes` bytes from shared memory to dst: whole words
// where dst is aligned, single bytes at the ends.
__device__ __forceinline__ void copy_out(uint8_t* dst, const uint8_t* src, int bytes) {
    const int head = min(bytes, (int)((4 - ((uintptr_t)dst & 3)) & 3)), words = (bytes - head) >> 2;
    const int t = threadIdx.x;
    for (int i = t; i < words; i += kMeshWork) {
        const uint8_t* p = src + head + 4 * i;
        *reinterpret_cast<uint32_t*>(dst + head + 4 * i) =
            (uint32_t)p[0] | (uint32_t)p[1] << 8 | (uint32_t)p[2] << 16 | (uint32_t)p[3] << 24;
    }
    const int tail = bytes - head - 4 * words;
    if (t < head) dst[t] = src[t];
    if (t < tail) dst[head + 4 * words + t] = src[head + 4 * words + t];
}

// The triangles.  One voxel per thread and its triangles one after another
// left most lanes idle and wrote 4 bytes every 12 (10 800 blocks, 880 000
// triangles: 211 us).  The block's triangles are listed from its rows' bits and
// its vertices are dealt to its threads: 95 us (116 with every voxel classified
// again, the tables in constant memory and the region's indices recomputed).
__global__ void __launch_bounds__(kMeshThreads, kMeshCtas)
    k_mesh_emit(MapView m, const unsigned long long* offsets, unsigned long long cap, float* V, float* N, uint8_t* C) {
    __shared__ MeshSmem s;
    __shared__ EmitSmem em;
    const int n = min(m.ctr->n_alloc, m.NS), t = threadIdx.x;
    const Region g = region_of(t);
    if (t < 64) reinterpret_cast<uint32_t*>(s.ntri)[t] = reinterpret_cast<const uint32_t*>(c_ntri)[t];
    if (t < 256) reinterpret_cast<uint4*>(em.table)[t] = reinterpret_cast<const uint4*>(c_tri)[t];
    walk_blocks(m, n, s, [&](int blk, int buf) {
        const unsigned long long first = offsets[blk];
        const int total = (int)min(offsets[blk + 1] - first, first < cap ? cap - first : 0ull);
        if (total == 0) return;   // uniform: no surface in this block, or no room left
        stage_block<true>(m, g, s, em.rgb, buf);
        // list the triangles in voxel order: row by row (thread t < 64: row
        // (t & 7, t >> 3)), the rows before this one's counted by a prefix
        // over both warps (warp 1 counts warp 0's rows again)
        if (t < 64) {
            const int lane = t & 31;
            auto count = [&](const CubeRow& c) {
                int nt = 0;
                for (uint32_t k = c.mask; k; k &= k - 1) nt += s.ntri[cube_case(c, __ffs(k) - 1)];
                __syncwarp();
                return nt;
            };
            const CubeRow c = cube_row(s, t & 7, t >> 3);
            const int nt = count(c);
            int o = nt;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, o, d);
                if (lane >= d) o += y;
            }
            o -= nt;
            if (t >= 32) o += __reduce_add_sync(0xffffffffu, count(cube_row(s, lane & 7, lane >> 3)));
            for (uint32_t k = c.mask; k; k &= k - 1) {
                const int x = __ffs(k) - 1, vx = 8 * t + x, ci = cube_case(c, x), nc = s.ntri[ci];
                em.cubes[vx] = (uint8_t)ci;
                for (int j = 0; j < nc; ++j) em.tri[o + j] = (uint16_t)(vx | j << 9);
                o += nc;
            }
        }
        work_barrier();
        const int3 b8 = make_int3(s.pos[buf].x * 8, s.pos[buf].y * 8, s.pos[buf].z * 8);
        for (int v0 = 0; v0 < 3 * total; v0 += kMeshWork) {
            const int cnt = min(kMeshWork, 3 * total - v0);
            if (t < cnt) {
                const int id = v0 + t, tr = em.tri[id / 3], vx = tr & 511;
                edge_vertex(s, em.rgb, vx & 7, (vx >> 3) & 7, vx >> 6, b8,
                            em.table[em.cubes[vx]][3 * (tr >> 9) + id % 3], m.g.voxel_size, em.v + 3 * t,
                            em.n + 3 * t, em.c + 3 * t);
            }
            work_barrier();
            const size_t o = (size_t)(first * 3 + v0) * 3;
            for (int i = t; i < 3 * cnt; i += kMeshWork) {
                V[o + i] = em.v[i];
                N[o + i] = em.n[i];
            }
            copy_out(C + o, em.c, 3 * cnt);
            work_barrier();
        }
    });
}

size_t mesh_scratch_bytes(int n_blocks) { return 8 * ((size_t)n_blocks + 2) + 8 * (size_t)n_blocks; }

// Mesh of the map: *total = triangles found (all of them, also beyond `cap`);
// the first min(total, cap) are written when V, N and C are given.  scratch:
// mesh_scratch_bytes of the pool, {total, offsets, counts}.  The kernels read
// the number of blocks on the device.  Synchronous on `st`.
int launch_mesh(const MapView& m, void* scratch, float* V, float* N, uint8_t* C, unsigned long long cap,
                unsigned long long* total, cudaStream_t st) {
    *total = 0;
    const int rc = ensure_tables();
    if (rc != FB_OK) return rc;
    unsigned long long* const sum = (unsigned long long*)scratch;
    unsigned long long* const offsets = sum + 1;
    uint2* const counts = (uint2*)(offsets + m.NS + 1);
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return FB_ECUDA;
    const int grid = sms * kMeshCtas;
    k_mesh_count<<<grid, kMeshThreads, 0, st>>>(m, counts);
    k_mesh_scan<<<1, 1024, 0, st>>>(m, counts, offsets, sum);
    if (V && N && C && cap > 0) k_mesh_emit<<<grid, kMeshThreads, 0, st>>>(m, offsets, cap, V, N, C);
    const cudaError_t le = cudaGetLastError();
    unsigned long long tot = 0;
    const cudaError_t ce = cudaMemcpyAsync(&tot, sum, sizeof tot, cudaMemcpyDeviceToHost, st);
    const cudaError_t se = cudaStreamSynchronize(st);
    if (le != cudaSuccess || ce != cudaSuccess || se != cudaSuccess) {
        fb_set_error_text(cudaGetErrorString(le != cudaSuccess ? le : (ce != cudaSuccess ? ce : se)));
        return FB_ECUDA;
    }
    *total = tot;
    return FB_OK;
}

}  // namespace fb

extern "C" {

int fb_mesh_case_table(int8_t* tri, int32_t* counts) {
    if (!tri || !counts) return FB_EINVAL;
    int8_t t[256][16];
    int n[256];
    if (fb::build_tables(t, n) != FB_OK) return FB_EINVAL;
    std::memcpy(tri, t, sizeof t);
    for (int i = 0; i < 256; ++i) counts[i] = n[i];
    return FB_OK;
}

int fb_write_ply(const char* path, const float* vertex, const float* normal, const uint8_t* color,
                 uint64_t no_triangles) {
    if (!path || (no_triangles && (!vertex || !normal || !color))) return FB_EINVAL;
    FILE* f = std::fopen(path, "wb");
    if (!f) {
        fb_set_error_text("fb_write_ply: cannot open the file");
        return FB_EINVAL;
    }
    std::vector<char> buf(1 << 22);
    setvbuf(f, buf.data(), _IOFBF, buf.size());
    const unsigned long long nv = (unsigned long long)no_triangles * 3;
    std::fprintf(f,
                 "ply\nformat ascii 1.0\nelement vertex %llu\nproperty float x\nproperty float y\n"
                 "property float z\nproperty float nx\nproperty float ny\nproperty float nz\n"
                 "property uchar red\nproperty uchar green\nproperty uchar blue\nelement face %llu\n"
                 "property list uchar uint vertex_indices\nend_header\n",
                 nv, (unsigned long long)no_triangles);
    for (unsigned long long i = 0; i < nv; ++i)
        std::fprintf(f, "%g %g %g %g %g %g %d %d %d\n", vertex[3 * i], vertex[3 * i + 1], vertex[3 * i + 2],
                     normal[3 * i], normal[3 * i + 1], normal[3 * i + 2], (int)color[3 * i], (int)color[3 * i + 1],
                     (int)color[3 * i + 2]);
    for (unsigned long long i = 0; i < (unsigned long long)no_triangles; ++i)
        std::fprintf(f, "3 %llu %llu %llu\n", 3 * i, 3 * i + 1, 3 * i + 2);
    const bool ok = std::ferror(f) == 0;
    if (std::fclose(f) != 0 || !ok) {
        fb_set_error_text("fb_write_ply: write failed");
        return FB_EINVAL;
    }
    return FB_OK;
}

}  // extern "C"
