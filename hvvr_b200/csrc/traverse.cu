// traverse.cu - tile-frustum BVH traversal on the GPU.
//
// The reference's two-level CPU traversal (cullThread, libraries/hvvr/raycaster/traversal.cpp:99-190):
//   blockCullKernel: traverseBlocks + BlockFrame::sort per 8192-sample block frustum
//                    (libraries/hvvr/raycaster/traverse_avx.h:293-410), one CTA each;
//   tileTreeKernel, tileTreeHugeKernel: traverseTiles per 128-sample tile frustum, starting from its
//                    block's sorted stack (traverse_avx.h:412-527), emitting the tile's triangle list:
//                    the nodes visited breadth first, the list's order recovered afterwards;
//   tileCullKernel:  the same as the reference runs it, node by node with a sorted stack, one warp per
//                    tile: what the breadth-first cull leaves (above 8,192 visits, bounds that do not
//                    nest) and callers that set the stack's size (tile_stack_entries).
// All rebuild the world-space frustum of Frustum::Frustum (traverse_avx.cpp:22-211) from the
// camera-space corner rays and the camera matrix (frustumTransform, traversal.h:38-47).
//
// In one sequential node visit lane l loads word l of the 128-byte node (one coalesced row) and serves one
// test of one child, whose six bounds it receives by shuffle (LaneTest). Ballots fold the per-lane results
// into the reference's 4-bit child masks. The arithmetic per test is the reference's lane arithmetic in every
// kernel (explicit fmaf where it uses _mm256_fmadd_ps, IEEE single ops elsewhere), so the lists are its lists.
#include <algorithm>
#include <mutex>

#include "../../include/hvvr_c.h"
#include "dev_common.cuh"

namespace hvb {

namespace {

constexpr unsigned kFull = 0xffffffffu;

#ifdef HVVR_VISIT_CLOCKS
// Profiling build only (make -C hvvr_b200/csrc visit-clocks): per global tile, the SM cycles of
// its tile-cull node visits split into phases, plus its visit count, read back through
// hvvr_dbg_visit_clocks. The counters cost registers and instructions of their own, so the
// phases' shares are what this build measures, not the production kernel's absolute times.
constexpr uint32_t kVisitClockTiles = 1u << 17;
enum : uint32_t {
    kVcRow,    // waiting for the node's row (loaded during the previous visit)
    kVcTest,   // child-row loads issued, child boxes shuffled, frustum plane/projection tests
    kVcLeaf,   // refine tests of passing leaf slots and recording their triangle ranges
    kVcInsert, // sorted insertion of two or more internal children
    kVcNext,   // choosing the next node (one child, an inserted child, or a pop)
    kVcTail,   // after the last visit: expanding the buffered ranges into the tile's list
    kVcPhases
};
__device__ unsigned long long gVisitClocks[kVisitClockTiles][kVcPhases + 1];
#define VISIT_MARK(phase, dep)                                                                                         \
    do {                                                                                                               \
        const long long t_ = phaseClock(dep);                                                                          \
        vcAcc[phase] += t_ - vcLast;                                                                                   \
        vcLast = t_;                                                                                                   \
    } while (0)
#else
#define VISIT_MARK(phase, dep) do { } while (0)
#endif

struct SmemFrustum {
    float tpLo[4][3], tpHi[4][3], w[4];
    float proj[3][8];
    float edge[12][3];
    float minF[12], maxF[12];
    int distIdx;
    int degenerate;
};

// Lane layout (child-major): lane l serves child c = l >> 3 and test slot j = l & 7. Slots
// 0-3 are the four frustum planes, 4-6 the x/y/z projection overlaps, 7 always passes; so
// child c passes testBVHNodeChildren when byte c of the ballot is 0xFF. For the refine, slot j
// tests edge axis j and, for j < 4, also edge axis 8 + j; child c is rejected when byte c of
// that ballot is nonzero.
struct LaneTest {
    float c0, c1, c2, c3, c4, c5, c6; // plane slots: lo xyz, hi xyz, w; projection slots: c0 = max side, c1 = -min side
    int kind;                         // 0 plane, 1 projection, 2 always pass
    int axis;                         // projection axis
    float e0x, e0y, e0z, mn0, mx0;
    float e1x, e1y, e1z, mn1, mx1;
    bool has1;
};

// Frustum::Frustum on world-space rays, computed cooperatively by one warp.
__device__ void buildFrustum(const Rays4& cr, const Mat4& M, SmemFrustum& f) {
    F3 o[4], d[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        o[i] = xformPoint(M, f3(cr.o[i][0], cr.o[i][1], cr.o[i][2]));
        d[i] = xformDir(M, f3(cr.d[i][0], cr.d[i][1], cr.d[i][2]));
    }
    const uint32_t lane = laneId();
    const bool inf0 = isinf(o[0].x);
    if (lane < 4) {
        const int p = int(lane);
        F3 n = f3(0.0f, 0.0f, 0.0f);
        float w = -INFINITY;
        if (!inf0) {
            n = cross3(d[p], d[(p + 1) & 3]);
            w = dot3(o[p], n);
        }
        const float c[3] = {n.x, n.y, n.z};
#pragma unroll
        for (int a = 0; a < 3; a++) {
            f.tpLo[p][a] = c[a] < 0.0f ? c[a] : 0.0f;
            f.tpHi[p][a] = c[a] > 0.0f ? -c[a] : 0.0f;
        }
        f.w[p] = w;
        if (p == 0) f.degenerate = (w == -INFINITY) ? 1 : 0;
    } else if (lane < 16) {
        const int e = int(lane) - 4, i = e / 3, k = e % 3;
        const F3 axis = f3(k == 0 ? 1.0f : 0.0f, k == 1 ? 1.0f : 0.0f, k == 2 ? 1.0f : 0.0f);
        const F3 ed = cross3(d[i], axis);
        f.edge[e][0] = ed.x;
        f.edge[e][1] = ed.y;
        f.edge[e][2] = ed.z;
        float mn = FLT_MAX, mx = -FLT_MAX;
#pragma unroll
        for (int p = 0; p < 4; p++) {
            const float d0 = fmaf(ed.x, o[p].x, fmaf(ed.y, o[p].y, ed.z * o[p].z));
            mn = mn < d0 ? mn : d0;
            mx = mx > d0 ? mx : d0;
            const float d1 = fmaf(ed.x, d[p].x, fmaf(ed.y, d[p].y, ed.z * d[p].z));
            const float a = d1 + .000001f, b = d1 - .000001f;
            const float amin = a < 0.0f ? a : 0.0f;
            const float bmax = b > 0.0f ? b : 0.0f;
            mn = amin * FLT_MAX + mn;
            mx = bmax * FLT_MAX + mx;
        }
        f.minF[e] = mn;
        f.maxF[e] = mx;
    } else if (lane < 19) {
        const int a = int(lane) - 16;
        float lanev[8];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float oc = a == 0 ? o[i].x : (a == 1 ? o[i].y : o[i].z);
            const float dc = a == 0 ? d[i].x : (a == 1 ? d[i].y : d[i].z);
            const float nd0 = -dc, nd1 = -(-dc);
            const float m0 = (0.0f > nd0) ? 0.0f : nd0;
            const float m1 = (0.0f > nd1) ? 0.0f : nd1;
            lanev[i] = -oc + FLT_MAX * m0;
            lanev[4 + i] = -(-oc) + FLT_MAX * m1;
        }
        float y[8];
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float p0 = lanev[4 * h + i], p1 = lanev[4 * h + (i ^ 2)];
                y[4 * h + i] = p0 > p1 ? p0 : p1;
            }
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float p0 = y[4 * h + i], p1 = y[4 * h + (i ^ 1)];
                f.proj[a][4 * h + i] = -(p0 > p1 ? p0 : p1);
            }
    } else if (lane == 19) {
        F3 avg = f3(0.0f, 0.0f, 0.0f);
#pragma unroll
        for (int p = 0; p < 4; p++) avg = avg + d[p];
        int idx;
        if (fabsf(avg.x) > fabsf(avg.y)) {
            if (fabsf(avg.x) > fabsf(avg.z)) idx = avg.x < 0 ? 0 : 1;
            else idx = avg.z < 0 ? 4 : 5;
        } else {
            if (fabsf(avg.y) > fabsf(avg.z)) idx = avg.y < 0 ? 2 : 3;
            else idx = avg.z < 0 ? 4 : 5;
        }
        f.distIdx = idx;
    }
    __syncwarp();
}

// blockTransformAndCullTask's cull of a tile frustum (libraries/hvvr/raycaster/render.cpp:270-279,
// 314-338): culled when all four corner rays, at their origin and 10000 units out, lie beyond
// one of the planes. Evaluated by every lane on the same world-space rays.
__device__ bool tileCulled(const Rays4& cr, const Mat4& M, const float (&pl)[4][4]) {
    F3 o[4], d[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        o[i] = xformPoint(M, f3(cr.o[i][0], cr.o[i][1], cr.o[i][2]));
        d[i] = xformDir(M, f3(cr.d[i][0], cr.d[i][1], cr.d[i][2]));
    }
    bool culled = false;
#pragma unroll
    for (int p = 0; p < 4; p++) {
        const F3 n = f3(pl[p][0], pl[p][1], pl[p][2]);
        const float dist = pl[p][3];
        bool allout = true;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            allout = allout && dot3(n, o[i]) > dist;
            allout = allout && dot3(n, o[i] + d[i] * 10000.0f) > dist;
        }
        culled = culled || allout;
    }
    return culled;
}

__device__ LaneTest loadLaneTest(const SmemFrustum& f) {
    LaneTest t;
    const uint32_t lane = laneId();
    const int c = int(lane >> 3), j = int(lane & 7);
    t.c0 = t.c1 = t.c2 = t.c3 = t.c4 = t.c5 = t.c6 = 0.0f;
    t.axis = 0;
    if (j < 4) {
        t.kind = 0;
        t.c0 = f.tpLo[j][0]; t.c1 = f.tpLo[j][1]; t.c2 = f.tpLo[j][2];
        t.c3 = f.tpHi[j][0]; t.c4 = f.tpHi[j][1]; t.c5 = f.tpHi[j][2];
        t.c6 = f.w[j];
    } else if (j < 7) {
        t.kind = 1;
        t.axis = j - 4;
        t.c0 = f.proj[j - 4][c];
        t.c1 = f.proj[j - 4][4 + c];
    } else {
        t.kind = 2;
    }
    t.e0x = f.edge[j][0]; t.e0y = f.edge[j][1]; t.e0z = f.edge[j][2];
    t.mn0 = f.minF[j]; t.mx0 = f.maxF[j];
    t.has1 = j < 4;
    const int e1 = t.has1 ? 8 + j : j;
    t.e1x = f.edge[e1][0]; t.e1y = f.edge[e1][1]; t.e1z = f.edge[e1][2];
    t.mn1 = f.minF[e1]; t.mx1 = f.maxF[e1];
    return t;
}

struct ChildBox {
    float xM, xN, yM, yN, zM, zN;
};

__device__ __forceinline__ ChildBox childBox(float v) {
    const uint32_t c = laneId() >> 3;
    ChildBox b;
    b.xM = __shfl_sync(kFull, v, c);
    b.xN = __shfl_sync(kFull, v, 4 + c);
    b.yM = __shfl_sync(kFull, v, 8 + c);
    b.yN = __shfl_sync(kFull, v, 12 + c);
    b.zM = __shfl_sync(kFull, v, 16 + c);
    b.zN = __shfl_sync(kFull, v, 20 + c);
    return b;
}

// Bit c set where byte c of m is all ones / nonzero. Per byte, (b & 0x7f) + 0x7f sets the byte's
// high bit exactly when its low seven bits are not all zero and never carries into the next byte
// (at most 0xfe), so the byte tests are exact; the multiply gathers bits 7, 15, 23, 31 into bits
// 21-24 (the partial products land on distinct bits, so nothing carries).
__device__ __forceinline__ uint32_t gatherByteFlags(uint32_t z) { return (((z >> 7) * 0x204081u) >> 21) & 0xfu; }
__device__ __forceinline__ uint32_t bytesAllOnes(uint32_t m) {
    const uint32_t s = (~m & 0x7f7f7f7fu) + 0x7f7f7f7fu; // high bit: the byte of ~m has a low bit set
    return gatherByteFlags(~s & m & 0x80808080u);
}
__device__ __forceinline__ uint32_t bytesNonZero(uint32_t m) {
    const uint32_t s = (m & 0x7f7f7f7fu) + 0x7f7f7f7fu;
    return gatherByteFlags((s | m) & 0x80808080u);
}

// Frustum::testBVHNodeChildren (traverse_avx.h:104-164)
__device__ __forceinline__ uint32_t testChildren(const ChildBox& b, const LaneTest& t) {
    const float lo = fmaf(t.c0, b.xM, fmaf(t.c1, b.yM, t.c2 * b.zM));
    const float hi = fmaf(t.c3, b.xN, fmaf(t.c4, b.yN, t.c5 * b.zN));
    const bool planePass = (lo + hi) <= t.c6;
    const float am = t.axis == 0 ? b.xM : (t.axis == 1 ? b.yM : b.zM);
    const float an = t.axis == 0 ? b.xN : (t.axis == 1 ? b.yN : b.zN);
    const bool projPass = (am >= t.c0) && (an >= t.c1);
    const bool pass = t.kind == 0 ? planePass : (t.kind == 1 ? projPass : true);
    return bytesAllOnes(__ballot_sync(kFull, pass));
}

// The reference adds +0.0f to each selected bound (turning -0 into +0); that only changes the
// sign of a zero product or sum, which no comparison below can see, so it is left out.
__device__ __forceinline__ bool edgeReject(const ChildBox& b, float ex, float ey, float ez, float mn, float mx) {
    const bool px = ex > 0.0f, py = ey > 0.0f, pz = ez > 0.0f;
    const float pX = px ? b.xM : -b.xN, nX = px ? -b.xN : b.xM;
    const float pY = py ? b.yM : -b.yN, nY = py ? -b.yN : b.yM;
    const float pZ = pz ? b.zM : -b.zN, nZ = pz ? -b.zN : b.zM;
    const float maxBox = fmaf(ex, pX, fmaf(ey, pY, ez * pZ));
    const float minBox = fmaf(ex, nX, fmaf(ey, nY, ez * nZ));
    return (maxBox < mn) || (mx < minBox);
}

// edgeReject for an edge axis with a zero component, without that component's (zero) product: e.x and
// e.y are the other two components, e.z and e.w the frustum's range along the axis
__device__ __forceinline__ bool edgeReject2(float aM, float aN, float bM, float bN, float4 e) {
    const bool pa = e.x > 0.0f, pb = e.y > 0.0f;
    const float maxBox = fmaf(e.x, pa ? aM : -aN, e.y * (pb ? bM : -bN));
    const float minBox = fmaf(e.x, pa ? -aN : aM, e.y * (pb ? -bN : bM));
    return (maxBox < e.z) | (e.w < minBox);
}

// Frustum::testBVHNodeChildrenRefine (traverse_avx.h:166-217): mask of rejected children
__device__ __forceinline__ uint32_t refineReject(const ChildBox& b, const LaneTest& t) {
    const bool rej0 = edgeReject(b, t.e0x, t.e0y, t.e0z, t.mn0, t.mx0);
    const bool rej1 = edgeReject(b, t.e1x, t.e1y, t.e1z, t.mn1, t.mx1);
    return bytesNonZero(__ballot_sync(kFull, rej0 || (t.has1 && rej1)));
}

// Number of consecutive stack entries, from position top-1 downwards, for which pred holds.
// Equivalent to the reference's serial shift loop; the guard band below position 0 stops it.
template <class Pred>
__device__ __forceinline__ uint32_t shiftCount(uint32_t top, Pred pred) {
    const uint32_t lane = laneId();
    uint32_t k = 0;
    for (;;) {
        const int p = int(top) - 1 - int(k) - int(lane);
        const bool pr = (p >= 0) && pred(uint32_t(p));
        const uint32_t b = __ballot_sync(kFull, pr);
        const uint32_t run = (b == kFull) ? 32u : uint32_t(__ffs(~b) - 1);
        k += run;
        if (run < 32u || k >= top) return k < top ? k : top;
    }
}

// a float's order under the denormals-are-zero comparison, as an unsigned integer above 0 (NaN excepted)
__device__ __forceinline__ uint32_t orderKey(float v) {
    uint32_t u = __float_as_uint(v);
    if ((u & 0x7f800000u) == 0) u = 0;
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

constexpr int kBlockWarps = 8;

// A block's traversal (traverseBlocks): entries are nodes still to be visited, and groups of passing
// leaf slots. The reference's stack is sorted by tDelta, the newest on top among equal ones; here the
// entries lie in any order with that order's key and their age, and the top is searched for.
struct BlockSmem {
    SmemFrustum f;
    uint32_t key[kBlockStack], seq[kBlockStack]; // order of the stack: (key, seq) ascending from the bottom; key 0: unused
    uint32_t delta[kBlockStack];                 // tDelta, or the leaf mask (at most 15)
    float tMin[kBlockStack];
    uint32_t node[kBlockStack];
    // a tested node's passing children: mask of leaf slots | mask of internal children << 4 (kUntested until
    // then), and the latter's tDelta, tMin and index
    uint32_t pass[kBlockStack];
    float childDelta[kBlockStack][4], childMin[kBlockStack][4];
    uint32_t child[kBlockStack][4];
    uint32_t work[kBlockWarps], workCount; // entries to test now; none: the traversal has ended
    uint32_t rank[kBlockStack];
    uint32_t unused[kBlockStack], used; // unused[used..]: the unused entries
};
constexpr uint32_t kUntested = 0xffffffffu;

// the view of a global block (blocks of one view are consecutive)
__device__ __forceinline__ const ViewDev& viewOfBlock(const ViewDev* __restrict__ views,
                                                      const uint32_t* __restrict__ blockView, uint32_t viewCount,
                                                      uint32_t blk) {
    return views[viewCount == 1 ? 0u : __ldg(blockView + blk)];
}

// A block walks up to a few hundred dependent node visits, each of which waits for its node's row
// if it misses L2; so the CTAs past the block-cull CTAs first bring every scene's node array into
// L2 (bulk prefetches of 4 KiB, issued at once; the traversing warps meet lines in flight or
// resident, and so do the tile culls that follow).
constexpr uint32_t kPrefetchCtas = 32, kPrefetchChunk = 4096;

__device__ void prefetchSceneNodes(const FrameDev& fr, uint32_t cta) {
    const uint32_t tid = cta * blockDim.x + threadIdx.x, threads = kPrefetchCtas * blockDim.x;
    for (uint32_t vi = 0; vi < fr.viewCount; vi++) {
        const ViewDev& V = fr.views[vi];
        // whole 128-byte nodes of a 128-byte-aligned array: every chunk starts 16-byte aligned and
        // its size is a multiple of 16
        const size_t bytes = size_t(V.prefetchNodes) * sizeof(Node);
        const char* base = reinterpret_cast<const char*>(V.nodes);
        for (size_t off = size_t(tid) * kPrefetchChunk; off < bytes; off += size_t(threads) * kPrefetchChunk) {
            const uint32_t n = uint32_t(bytes - off < kPrefetchChunk ? bytes - off : kPrefetchChunk);
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(base + off), "r"(n) : "memory");
        }
    }
}

// One CTA per block. The traversal visits the entry on top of its stack until 60 entries are on it or
// only leaf groups are left, so the visits depend on each other; but what a visit costs is the tests of
// its node's children, and those depend on nothing. So the first warp takes visits from the stack as
// long as their nodes are tested, then the eight warps test eight of the waiting nodes, the top among
// them (the others are visited soon, or stay as the block's stack). One warp that tested and visited
// node by node took about 1 us a visit, up to 178 visits a block. The stage (with its memsets), before and
// after, one B200: 57k triangles 640 x 480 102 and 55 us; 1M stereo 103 and 69 us, from another pose 147 and
// 87; 160 x 120 63 and 32 us. What bounds it now: the chain of visits, about 300 cycles each.
__global__ void __launch_bounds__(kBlockWarps * 32) blockCullKernel(FrameDev fr) {
    __shared__ BlockSmem s;
    if (blockIdx.x >= fr.blocks) {
        prefetchSceneNodes(fr, blockIdx.x - fr.blocks);
        return;
    }
    const uint32_t warp = threadIdx.x >> 5, lane = laneId();
    const uint32_t gblk = blockIdx.x;
    const ViewDev& V = viewOfBlock(fr.views, fr.blockView, fr.viewCount, gblk);
    const uint32_t blk = gblk - V.blockStart;
    const float* rows = reinterpret_cast<const float*>(V.nodes);
    if (warp == 0) buildFrustum(V.blockRays[blk], V.M, s.f);
    else if (warp == 1)
        for (uint32_t i = lane; i < kBlockStack; i += 32) {
            s.rank[i] = 0;
            s.unused[i] = i;
            s.key[i] = i ? 0u : ~0u; // (entry 0: the root)
            s.seq[i] = 0;
            s.delta[i] = ~0u;
            s.tMin[i] = 0.0f;
            s.node[i] = 0;
            s.pass[i] = kUntested;
        }
    __syncthreads();
    if (s.f.degenerate) {
        if (threadIdx.x == 0) V.blockSizes[blk] = 0;
        return;
    }
    const LaneTest t = loadLaneTest(s.f);
    const int distIdx = s.f.distIdx, maxIdx = distIdx & ~1;
    // (the first warp's, the same on every lane) entries in use, the next one's age
    uint32_t used = 1, seq = 1;
    bool root = true;
    for (;;) {
        if (warp == 0) {
            uint32_t top = 0, k0, k1;
            bool done = false;
            for (;;) {
                k0 = s.key[lane];
                k1 = s.key[lane + 32];
                const uint32_t best = __reduce_max_sync(kFull, max(k0, k1));
                uint32_t b0 = __ballot_sync(kFull, k0 == best), b1 = __ballot_sync(kFull, k1 == best);
                done = best == 0; // no entries (keys are above 0)
                if (done) break;
                if ((b0 & (b0 - 1u)) | (b1 & (b1 - 1u)) || (b0 && b1)) {
                    const uint32_t q0 = k0 == best ? s.seq[lane] + 1u : 0u, q1 = k1 == best ? s.seq[lane + 32] + 1u : 0u;
                    const uint32_t newest = __reduce_max_sync(kFull, max(q0, q1));
                    b0 = __ballot_sync(kFull, q0 == newest);
                    b1 = __ballot_sync(kFull, q1 == newest);
                }
                top = b0 ? uint32_t(__ffs(b0) - 1) : uint32_t(__ffs(b1) + 31);
                const uint32_t pass = s.pass[top];
                done = !root && (used >= kBlockStack - 4 || s.delta[top] <= 0xfu);
                if (done || pass == kUntested) break;
                // visit it: its leaf group, then its children in slot order
                root = false;
                const uint32_t leaf = pass & 15u, inner = pass >> 4, group = leaf ? 1u : 0u, count = group + __popc(inner);
                if (lane < count) {
                    const uint32_t e = s.unused[used + lane];
                    uint32_t d = leaf, nd = s.node[top];
                    float tm = s.tMin[top];
                    if (lane >= group) {
                        uint32_t m = inner;
                        if (lane - group > 0) m &= m - 1u;
                        if (lane - group > 1) m &= m - 1u;
                        if (lane - group > 2) m &= m - 1u;
                        const uint32_t k = uint32_t(__ffs(m) - 1);
                        d = __float_as_uint(s.childDelta[top][k]);
                        tm = s.childMin[top][k];
                        nd = s.child[top][k];
                    }
                    s.key[e] = orderKey(__uint_as_float(d));
                    s.seq[e] = seq + lane;
                    s.delta[e] = d;
                    s.tMin[e] = tm;
                    s.node[e] = nd;
                    s.pass[e] = kUntested;
                }
                __syncwarp();
                seq += count;
                used += count - 1u;
                if (lane == 0) {
                    s.key[top] = 0;
                    s.unused[used] = top;
                }
                __syncwarp();
            }
            if (done) {
                if (lane == 0) {
                    s.workCount = 0;
                    s.used = used;
                }
            } else {
                // the top, and others that wait to be tested (leaf groups do not)
                const bool w0 = k0 && s.pass[lane] == kUntested && s.delta[lane] > 0xfu && lane != top;
                const bool w1 = k1 && s.pass[lane + 32] == kUntested && s.delta[lane + 32] > 0xfu && lane + 32 != top;
                const uint32_t b0 = __ballot_sync(kFull, w0), b1 = __ballot_sync(kFull, w1);
                const uint32_t p0 = 1u + __popc(b0 & ((1u << lane) - 1u)), p1 = 1u + __popc(b0) + __popc(b1 & ((1u << lane) - 1u));
                if (w0 && p0 < kBlockWarps) s.work[p0] = lane;
                if (w1 && p1 < kBlockWarps) s.work[p1] = lane + 32;
                if (lane == 0) {
                    s.work[0] = top;
                    s.workCount = min(1u + __popc(b0) + __popc(b1), uint32_t(kBlockWarps));
                }
            }
        }
        __syncthreads();
        if (s.workCount == 0) break;
        if (warp < s.workCount) {
            const uint32_t e = s.work[warp], node = s.node[e];
            const float v = rows[size_t(node) * 32 + lane];
            const ChildBox cb = childBox(v);
            const uint32_t mask = testChildren(cb, t) & ~refineReject(cb, t);
            const uint32_t leafMask = __float_as_uint(__shfl_sync(kFull, v, 24));
            const uint32_t k = lane & 3u;
            const float tm = __uint_as_float(__float_as_uint(__shfl_sync(kFull, v, distIdx * 4 + k)) ^ 0x80000000u);
            const float hi = __shfl_sync(kFull, v, maxIdx * 4 + k), lo = __shfl_sync(kFull, v, (maxIdx + 1) * 4 + k);
            const uint32_t child = node + __float_as_uint(__shfl_sync(kFull, v, 26 + k));
            if (lane < 4) {
                s.childDelta[e][k] = hi + lo;
                s.childMin[e][k] = tm;
                s.child[e][k] = child;
            }
            if (lane == 0) s.pass[e] = (mask & leafMask) | ((mask & ~leafMask) << 4);
        }
        __syncthreads();
    }
    // BlockFrame::sort: by distance estimate, the closest on top; the stack's order among equal ones
    for (uint32_t h = 0; h < 2; h++) {
        const uint32_t i = lane + 32 * h, key = s.key[i], age = s.seq[i];
        if (!key) continue;
        const float mine = dazf(s.tMin[i]);
        uint32_t below = 0;
        for (uint32_t j = warp * 8; j < warp * 8 + 8; j++) {
            const float other = dazf(s.tMin[j]);
            const uint32_t otherKey = s.key[j];
            const bool first = otherKey < key || (otherKey == key && s.seq[j] < age);
            if (otherKey && (other > mine || (other == mine && first))) below++;
        }
        if (below) atomicAdd(&s.rank[i], below);
    }
    __syncthreads();
    if (threadIdx.x < kBlockStack && s.key[threadIdx.x]) {
        const uint32_t i = threadIdx.x, d = s.delta[i];
        V.blockStacks[size_t(blk) * kBlockStack + s.rank[i]] = StackEntry{s.tMin[i], d > 0xfu ? 0u : d, s.node[i]};
    }
    if (threadIdx.x == 0) V.blockSizes[blk] = s.used;
}

// per-warp tile traversal state; S = sorted-stack capacity
// passing leaf slots buffered per warp as triangle ranges before they are expanded into the list
constexpr uint32_t kRanges = 128;

template <uint32_t S>
struct TileSmemT {
    SmemFrustum f;
    float tMin[S];
    uint32_t mask[S];
    uint32_t node[S];
    alignas(16) uint32_t buf[kChunk];
    uint32_t rStart[kRanges], rLen[kRanges];
};

struct Emitter {
    uint32_t* pool;
    uint32_t* chunkNext;
    uint32_t poolChunks;
    uint32_t* counters;
    uint32_t first, prev, bufCount, stored, total;
    bool dead;
    uint32_t rc; // ranges buffered in rStart/rLen

    __device__ void flush(uint32_t* buf) {
        __syncwarp();
        uint32_t c = 0;
        if (laneId() == 0) c = atomicAdd(&counters[0], 1u);
        c = __shfl_sync(kFull, c, 0);
        if (c >= poolChunks) {
            if (laneId() == 0) atomicOr(&counters[1], kStatusPoolOverflow);
            dead = true;
            return;
        }
        const uint4 w = reinterpret_cast<const uint4*>(buf)[laneId()];
        reinterpret_cast<uint4*>(pool + size_t(c) * kChunk)[laneId()] = w;
        if (laneId() == 0 && prev != kNoChunk) chunkNext[prev] = c;
        if (prev == kNoChunk) first = c;
        prev = c;
        stored += bufCount;
        bufCount = 0;
        __syncwarp();
    }

    // Records the triangle ranges of the passing leaf slots of one node, in slot order (leaf
    // slot k covers [tri[k], tri[k+1]) = words 25+k, 26+k of the node; v holds word l of the
    // node in lane l). The entries are written out later by expand(), in the same order.
    template <uint32_t S>
    __device__ void addLeaves(TileSmemT<S>& s, float v, uint32_t leaf) {
        const uint32_t lane = laneId(), k = lane & 3u;
        const uint32_t t0 = __float_as_uint(__shfl_sync(kFull, v, 25 + k));
        const uint32_t t1 = __float_as_uint(__shfl_sync(kFull, v, 26 + k));
        const bool on = lane < 4 && ((leaf >> k) & 1u);
        if (on && t1 <= t0) atomicOr(&counters[1], kStatusBadLeaf);
        const bool emit = on && t1 > t0;
        const uint32_t b = __ballot_sync(kFull, emit);
        if (rc + 4 > kRanges) expand(s);
        if (emit) {
            const uint32_t pos = rc + __popc(b & ((1u << lane) - 1u));
            s.rStart[pos] = t0;
            s.rLen[pos] = t1 - t0;
        }
        rc += __popc(b);
        __syncwarp();
    }

    // Expands the buffered ranges into list entries (through buf, flushed to the pool per
    // chunk), 32 ranges at a time: lane r holds range r's start and the exclusive prefix of
    // the lengths, and each entry finds its range by a binary search over the lanes.
    template <uint32_t S>
    __device__ void expand(TileSmemT<S>& s) {
        const uint32_t lane = laneId();
        for (uint32_t r0 = 0; r0 < rc && !dead; r0 += 32) {
            const uint32_t r = r0 + lane;
            const uint32_t len = r < rc ? s.rLen[r] : 0u;
            const uint32_t start = r < rc ? s.rStart[r] : 0u;
            uint32_t inc = len;
#pragma unroll
            for (uint32_t o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(kFull, inc, o);
                if (lane >= o) inc += y;
            }
            const uint32_t n = __shfl_sync(kFull, inc, 31);
            const uint32_t excl = inc - len; // lanes past the last range hold n
            uint32_t done = 0;
            while (done < n && !dead) {
                const uint32_t m = min(n - done, kChunk - bufCount);
                for (uint32_t base = 0; base < m; base += 32) {
                    const uint32_t j = base + lane;
                    const uint32_t p = done + j;
                    uint32_t lo = 0;
#pragma unroll
                    for (uint32_t step = 16; step; step >>= 1) {
                        const uint32_t e = __shfl_sync(kFull, excl, lo + step);
                        if (e <= p) lo += step;
                    }
                    const uint32_t st = __shfl_sync(kFull, start, lo);
                    const uint32_t pre = __shfl_sync(kFull, excl, lo);
                    if (j < m) s.buf[bufCount + j] = st + (p - pre);
                }
                bufCount += m;
                done += m;
                total += m;
                if (bufCount == kChunk) flush(s.buf);
            }
        }
        rc = 0;
        __syncwarp();
    }
};

struct TileCullArgs {
    const ViewDev* views;
    const uint32_t* blockView;
    uint32_t viewCount;
    uint32_t* pool;
    uint32_t* chunkNext;
    uint32_t poolChunks;
    uint32_t* counters;    // [0] chunk allocator, [1] status
    const uint32_t* order; // global tile order for the queue (nullptr = natural order)
    uint32_t first;        // this launch culls order[first, first + count)
    uint32_t count;
    uint32_t* queue;       // work-queue head of this launch, zero at launch
    uint32_t* retry;       // tiles whose stack outgrew kTileStack, at retry[first + i]
    uint32_t* retryCount;  // number of such tiles, zero at launch
    uint32_t stackLimit;   // entries the main pass may use (<= kTileStack)
    uint32_t* ready;       // pipelined: ready slots, slot first + i for the i-th finished tile (else nullptr)
    uint32_t* readyTail;   // pipelined: finished tiles so far, zero at launch
    uint32_t persistent;   // 0: every warp culls one tile (the grid has a warp per tile), then exits
    const uint32_t* counts; // breadth-first cull: the large, and of those the huge, tiles at the front of the rate
                           // class's order (nullptr: none)
    uint32_t noHuge;       // 1: the huge are culled as the large are
    uint32_t* bigQueue;    // work-queue head of the large tiles, zero at launch
    void* giants;          // kGiantSlots stores in global memory (nullptr: none), and, zero at launch,
    uint32_t* giantSlots;  // those taken by the huge tiles' launch
    uint32_t* giantQueue;  // work-queue head of the retry pass's giant tiles

    __device__ uint32_t big() const { return counts ? min(__ldcg(counts), count) : 0u; }
    __device__ uint32_t huge() const { return counts && !noHuge ? min(__ldcg(counts + 1), count) : 0u; }
};

// traverseTiles for one tile of view V (tile = view-local index); returns the node visits.
// overflow: the sorted stack needed more than S entries; the tile's list is left empty.
template <uint32_t S>
__device__ uint32_t cullTile(const TileCullArgs& a, const ViewDev& V, uint32_t tile, TileSmemT<S>& s, bool& overflow) {
    overflow = false;
    const uint32_t lane = laneId();
    const Node* __restrict__ nodes = V.nodes;
    const uint32_t blk = tile / kTilesPerBlock;
    const uint32_t stackSize = V.blockSizes[blk];
    buildFrustum(V.tileRays[tile], V.M, s.f);
    if (V.hasCull && tileCulled(V.tileRays[tile], V.M, V.cull)) {
        if (lane == 0) V.tileLists[tile] = TileList{kNoChunk, 0};
        return 0;
    }
    if (stackSize == 0 || s.f.degenerate) {
        if (lane == 0) V.tileLists[tile] = TileList{kNoChunk, 0};
        return 0;
    }
    for (uint32_t i = lane; i < stackSize; i += 32) {
        const StackEntry e = V.blockStacks[size_t(blk) * kBlockStack + i];
        s.tMin[i] = e.tMin;
        s.mask[i] = e.mask;
        s.node[i] = e.node;
    }
    __syncwarp();
    const LaneTest t = loadLaneTest(s.f);
    const int distIdx = s.f.distIdx;
    Emitter em{a.pool, a.chunkNext, a.poolChunks, a.counters, kNoChunk, kNoChunk, 0, 0, 0, false, 0};
    uint32_t top = stackSize - 1;
    uint32_t node = s.node[top];
    uint32_t visits = 0;
    const float* rows = reinterpret_cast<const float*>(nodes);
    float v = rows[size_t(node) * 32 + lane];
#ifdef HVVR_VISIT_CLOCKS
    long long vcAcc[kVcPhases] = {0, 0, 0, 0, 0, 0};
    long long vcLast = phaseClock(node);
#endif
    for (;;) {
        ++visits;
        // The next visit is always one of this node's internal children or the stack entry
        // below the current one (a pop, or a push whose children all sort below it), so their
        // rows are loaded now and consumed at the end of the visit, hiding the load latency.
        const uint32_t leafMask = __float_as_uint(__shfl_sync(kFull, v, 24));
        VISIT_MARK(kVcRow, leafMask);
        uint32_t childNode[4];
        float vc[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            childNode[k] = node + __float_as_uint(__shfl_sync(kFull, v, 26 + k));
            vc[k] = ((leafMask >> k) & 1u) ? 0.0f : rows[size_t(childNode[k]) * 32 + lane];
        }
        const bool hasPop = top > 0;
        const uint32_t popNode = hasPop ? s.node[top - 1] : 0u;
        const float vp = hasPop ? rows[size_t(popNode) * 32 + lane] : 0.0f;
        const ChildBox cb = childBox(v);
        uint32_t mask = testChildren(cb, t);
        VISIT_MARK(kVcTest, mask);
        if (mask) {
            uint32_t leaf = mask & leafMask;
            if (leaf) {
                mask &= ~refineReject(cb, t);
                leaf = mask & leafMask;
                if (leaf) em.addLeaves(s, v, leaf);
                VISIT_MARK(kVcLeaf, em.rc);
                if (em.dead) break;
            }
            mask &= ~leafMask;
            if (mask && s.mask[top] == 0u) {
                int k = __ffs(mask) - 1;
                if (!(mask & (mask - 1))) {
                    // (child indices by shuffle: a register array indexed at run time would live
                    // in local memory)
                    node = node + __float_as_uint(__shfl_sync(kFull, v, 26 + k));
                    v = vc[0];
#pragma unroll
                    for (int q = 1; q < 4; q++)
                        if (q == k) v = vc[q];
                    VISIT_MARK(kVcNext, node);
                    continue;
                }
                // Insert all m >= 2 children at once. Keys are never NaN (a child that passes the
                // plane test has finite bounds), so the stack stays sorted, non-increasing from
                // bottom to top under the DAZ comparison, and the reference's one-at-a-time
                // insertion (shift entries with a smaller key up, place the child, newest above
                // equal keys) is equivalent to: an old entry moves up by the number of children
                // with a larger key; child i lands at
                //   top - #{old < key_i} + #{children with a larger key}
                //       + #{earlier children with an equal key}.
                const uint32_t m = __popc(mask);
                if (top + m >= (S == kTileStack ? a.stackLimit : S)) {
                    overflow = true;
                    break;
                }
                // the children in slot order (bit i of mask: child i is inserted); the reference
                // inserts them in slot order, so "earlier" in the tie rule is the earlier slot
                float ck[4], ckz[4];
                float maxKey = -INFINITY, minKey = INFINITY;
                uint32_t kmin = 0;
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    ck[i] = __uint_as_float(__float_as_uint(__shfl_sync(kFull, v, distIdx * 4 + i)) ^ 0x80000000u);
                    ckz[i] = dazf(ck[i]);
                    if ((mask >> i) & 1u) {
                        maxKey = fmaxf(maxKey, ckz[i]);
                        if (ckz[i] <= minKey) { minKey = ckz[i]; kmin = uint32_t(i); }
                    }
                }
                // old entries that move: those with a key below the largest child key (a top run).
                // Lane j holds entry top-1-j of a group of 32; the first group is read once both
                // to find the run and to move it, and the run continues into later groups only
                // when all 32 of the first move.
                uint32_t less[4] = {0u, 0u, 0u, 0u};
                auto moveGroup = [&](uint32_t j, bool act, float e, float ez, uint32_t em_, uint32_t en) {
                    const uint32_t p = top - 1 - j;
                    uint32_t d = 0;
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const bool valid = (mask >> i) & 1u;
                        d += (act && valid && ckz[i] > ez) ? 1u : 0u;
                        less[i] += __popc(__ballot_sync(kFull, act && valid && ez < ckz[i]));
                    }
                    __syncwarp();
                    if (act && d) { s.tMin[p + d] = e; s.mask[p + d] = em_; s.node[p + d] = en; }
                    __syncwarp();
                };
                uint32_t region;
                float oldTopKey; // key of the entry below the current one (when there is one)
                {
                    const bool inb = lane < top;
                    float e = 0.0f, ez = 0.0f;
                    uint32_t em_ = 0, en = 0;
                    if (inb) {
                        const uint32_t p = top - 1 - lane;
                        e = s.tMin[p]; em_ = s.mask[p]; en = s.node[p]; ez = dazf(e);
                    }
                    oldTopKey = __shfl_sync(kFull, ez, 0);
                    const uint32_t b = __ballot_sync(kFull, inb && ez < maxKey);
                    region = (b == kFull) ? 32u : uint32_t(__ffs(~b) - 1);
                    moveGroup(lane, lane < region, e, ez, em_, en);
                    if (region == 32u && top > 32u)
                        region = 32u + shiftCount(top - 32u, [&](uint32_t p) { return dazf(s.tMin[p]) < maxKey; });
                }
                for (uint32_t base = 32; base < region; base += 32) {
                    const uint32_t j = base + lane;
                    const bool act = j < region;
                    float e = 0.0f, ez = 0.0f;
                    uint32_t em_ = 0, en = 0;
                    if (act) { const uint32_t p = top - 1 - j; e = s.tMin[p]; em_ = s.mask[p]; en = s.node[p]; ez = dazf(e); }
                    moveGroup(j, act, e, ez, em_, en);
                }
                if ((mask >> lane) & 1u) { // lanes 0-3, one per inserted child
                    uint32_t pos = top - less[0];
                    float mine = ckz[0];
                    float rawk = ck[0];
                    uint32_t nd = childNode[0];
#pragma unroll
                    for (int i = 1; i < 4; i++)
                        if (uint32_t(i) == lane) { pos = top - less[i]; mine = ckz[i]; rawk = ck[i]; nd = childNode[i]; }
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        if (!((mask >> i) & 1u) || uint32_t(i) == lane) continue;
                        if (ckz[i] > mine || (ckz[i] == mine && uint32_t(i) < lane)) pos++;
                    }
                    s.tMin[pos] = rawk;
                    s.mask[pos] = 0u;
                    s.node[pos] = nd;
                }
                __syncwarp();
                const bool popNext = hasPop && oldTopKey < minKey;
                top += m - 1;
                VISIT_MARK(kVcInsert, top);
                // The new top entry is the next node: the old entry below the current one when its
                // key is below every child's (it moved up by m), else the child with the smallest
                // key, the last slot among equal ones (an old entry with an equal key stays below it).
                if (popNext) {
                    node = popNode;
                    v = vp;
                } else {
                    node = childNode[0];
                    v = vc[0];
#pragma unroll
                    for (uint32_t q = 1; q < 4; q++)
                        if (q == kmin) { node = childNode[q]; v = vc[q]; }
                }
                VISIT_MARK(kVcNext, node);
                continue;
            }
        }
        if (top == 0) break;
        --top;
        node = popNode;
        v = vp;
        VISIT_MARK(kVcNext, node);
    }
#ifdef HVVR_VISIT_CLOCKS
    vcLast = phaseClock(top);
#endif
    if (overflow) {
        if (lane == 0) V.tileLists[tile] = TileList{kNoChunk, 0};
        return visits;
    }
    if (!em.dead && em.rc) em.expand(s);
    if (!em.dead && em.bufCount) em.flush(s.buf);
    if (lane == 0) {
        if (em.prev != kNoChunk) a.chunkNext[em.prev] = kNoChunk;
        V.tileLists[tile] = TileList{em.first, em.dead ? em.stored : em.total};
    }
#ifdef HVVR_VISIT_CLOCKS
    VISIT_MARK(kVcTail, em.total);
    if (lane == 0 && V.tileStart + tile < kVisitClockTiles) {
        for (uint32_t k = 0; k < kVcPhases; k++) gVisitClocks[V.tileStart + tile][k] = uint64_t(vcAcc[k]);
        gVisitClocks[V.tileStart + tile][kVcPhases] = visits;
    }
#endif
    return visits;
}

// Publishes a finished tile to the concurrent shade: every thread's list writes are made visible
// device-wide before one releases the ready slot.
template <int W>
__device__ __forceinline__ void publishTile(const TileCullArgs& a, uint32_t gt, bool retry) {
    if (!a.ready) return;
    __threadfence();
    if constexpr (W == 1) __syncwarp();
    else __syncthreads();
    if ((W == 1 ? laneId() : threadIdx.x) == 0) {
        const uint32_t pos = atomicAdd(a.readyTail, 1u);
        const uint32_t val = gt | (retry ? kReadyRetry : 0u);
        asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(a.ready + a.first + pos), "r"(val) : "memory");
    }
}

// Persistent warps pull tiles from a queue (longest-first when an order is given), so a
// few long horizon tiles overlap with the rest instead of holding a CTA slot each. Non-persistent
// (a.persistent == 0): the grid has a warp per tile and each warp takes one tile from the same
// queue, so the tiles still start longest-first and every CTA ends with its tile.
// (W = 1: one warp per CTA, so a warp that runs out of tiles frees its registers at once; the
// bound asks for the 20 resident warps per SM that the wider CTAs reach)
template <int W>
__global__ void __launch_bounds__(W * 32, W == 1 ? 20 : 1) tileCullKernel(TileCullArgs a) {
    __shared__ TileSmemT<kTileStack> smem[W];
    const uint32_t warp = threadIdx.x >> 5, lane = laneId();
    TileSmemT<kTileStack>& s = smem[warp];
    // A launch that follows this one with programmatic serialization (the pipelined shade) may be
    // scheduled once every CTA of this grid has started: its CTAs wait for tiles that only this
    // grid's warps publish, so they must never keep a cull CTA from becoming resident.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    for (;;) {
        uint32_t w = 0;
        if (lane == 0) w = atomicAdd(a.queue, 1u);
        w = __shfl_sync(kFull, w, 0);
        if (w >= a.count) return;
        const uint32_t gt = a.order ? a.order[a.first + w] : a.first + w;
        const ViewDev& V = viewOfBlock(a.views, a.blockView, a.viewCount, gt / kTilesPerBlock);
        const uint32_t tile = gt - V.tileStart;
        __syncwarp();
        bool overflow;
        const uint32_t visits = cullTile(a, V, tile, s, overflow);
        if (lane == 0) {
            V.tileCost[tile] = visits;
            if (overflow) a.retry[a.first + atomicAdd(a.retryCount, 1u)] = gt;
        }
        publishTile<1>(a, gt, overflow);
        __syncwarp();
        if (!a.persistent) return;
    }
}

// ---------------------------------------------------------------- breadth-first tile cull
// traverseTiles without its serial chain of node visits. The traversal has no early out: it visits
// every node whose ancestors pass the tile's tests, and its sorted stack only decides the order in
// which the passing leaves' triangles enter the list. So the nodes are visited breadth first, eight
// per warp step (lane = node * 4 + child), and the order is recovered afterwards:
//
//   The stack pops the smallest key, newest first among equal keys, and a node with a single
//   passing child goes to it at once (an edge of key -infinity). For two visited nodes a and b with
//   lowest common ancestor L, a comes first when the largest key on the path from L to a is smaller
//   than the one on the path to b (the element that holds b's maximum cannot be popped while
//   anything on a's path is pending); with equal maxima, the first elements that hold them were
//   pushed when their parents were popped, and the one pushed later is popped first - so the order
//   of the parents, reversed (or the later slot, for siblings).
//   Child boxes nest, so keys do not fall along a path, and the nodes form connected components: a
//   component's head is a child of a node with several passing children, with a key above its
//   parent's component's; a child with an equal key, and a single child, belong to the parent's
//   component. A component is popped without interruption, in depth-first order, later slots first.
//   The block's stack entries are the roots; their keys may be measured along another axis than the
//   tile's, so a root's key takes part only in comparisons between different roots.
//
// Components with passing leaves are sorted by (largest key on the path, then compBefore), and a
// node's place is its component's start plus its depth-first offset. A tile that does not fit the
// store, or whose keys fall along a path (bounds that do not nest, NaN), is left to the sequential
// kernels, which give the same list for every input.
//
// What bounds it: issue and the barriers between generations (54% of the issue slots, ncu), with about
// 60 instructions per visit; eight warps per large tile and four CTAs (64 registers) per SM keep both
// short chains and enough warps. The sequential traversal is a chain of about 2,000 cycles per visit.
// The cull launch alone, before and after, one B200: 57k triangles 640 x 480, 229 and 81 us; 1M
// triangles 1280 x 720, 3,364 and 371 us; 1M triangles stereo 2 x 1080 x 1200, 2,511 and 978 us. With
// two CTAs of 128 registers per SM the last took 1,255 us.
constexpr uint32_t kTreeWarps = 8;
constexpr uint32_t kWarpNodes = 256;                       // visited nodes of a tile culled by one warp,
constexpr uint32_t kCtaNodes = kTreeWarps * kWarpNodes;    // of one culled by a CTA of 8 warps,
constexpr uint32_t kHugeWarps = 16, kHugeNodes = 8192;     // by a CTA of 16 warps that has an SM for itself,
constexpr uint32_t kGiantNodes = 32768;                    // and by such a CTA with a store in global memory
constexpr uint32_t kMaxGens = 64;
constexpr uint32_t kRetryStack = 4096;
constexpr uint32_t kMaxLeafRange = 65535;                  // longer leaf ranges are left to the sequential kernels

// A component is named by its head's store index.
template <uint32_t N>
struct TreeStore {
    static constexpr uint32_t kNodes = N, kSorted = N / 2;
    unsigned long long sortKey[kSorted]; // largest key on the path << 32 | component; later list staging
    uint32_t node[N];
    uint32_t key[N];        // order key of a component's head, 0 for a root's
    uint32_t meta[N];       // kMeta... below
    uint16_t first[N];      // first child; later the nodes in traversal order
    uint16_t comp[N];
    uint16_t size[N];       // nodes of the component at and below the node, then the depth-first offset
    uint16_t compSize[N];   // of heads; then the component's first position
};
// meta: a head's parent (bits 0-14), root index (15-20), whether its component has passing leaves
// (21); a node's passing leaf slots (22-25) and internal children (26-28); a root that stands for
// leaf slots only (29)
constexpr uint32_t kMetaParent = 0x7fffu, kMetaRoot = 15, kMetaLeafy = 1u << 21, kMetaSlots = 22, kMetaChildren = 26,
                   kMetaMasked = 1u << 29;
static_assert(kGiantNodes <= kMetaParent + 1, "parent index bits");
static_assert(sizeof(TreeStore<kWarpNodes>::sortKey) >= sizeof(SmemFrustum), "the frustum is built in the sort's memory");

struct TreeHead {
    float4 lo[4], hi[4];     // frustum planes: tpLo, w | tpHi
    float4 edge[12];         // edge axes, the two components that the cross product with an axis leaves; min, max
    uint32_t rootKey[kBlockStack];
    uint16_t gen[kMaxGens + 2]; // generation g is nodes [gen[g], gen[g + 1])
    uint32_t pushed[3];      // nodes pushed in a generation (in turn), kPushedBad added where the tile cannot be culled here
    uint32_t total, first, sorted;
    uint32_t warpSum[kHugeWarps];
};
constexpr uint32_t kPushedBad = 1u << 20;

struct TreeSmem {
    TreeHead head[kTreeWarps];
    union {
        TreeStore<kWarpNodes> warp[kTreeWarps];
        TreeStore<kCtaNodes> cta;
    };
    uint32_t item, spill;
};
struct HugeSmem {
    TreeHead head;
    union {
        TreeStore<kHugeNodes> cta;
        TileSmemT<kRetryStack> seq;
    };
    uint32_t item;
};

// whether component a is popped before component b (see above); called where the sort keys are equal
template <class S>
__device__ __noinline__ bool compBefore(const S& s, const uint32_t* rootKey, uint32_t a, uint32_t b) {
    bool flip = false;
    for (;;) {
        const uint32_t ma = s.meta[a], mb = s.meta[b], ka = s.key[a], kb = s.key[b];
        const uint32_t ra = (ma >> kMetaRoot) & 63u, rb = (mb >> kMetaRoot) & 63u;
        const bool sameRoot = ra == rb;
        const uint32_t ea = sameRoot ? ka : max(rootKey[ra], ka), eb = sameRoot ? kb : max(rootKey[rb], kb);
        if (ea != eb) return (ea < eb) != flip;
        if (!sameRoot) {
            // a root that holds its path's maximum was there from the start: below anything pushed
            // since, and roots in stack order
            const bool la = rootKey[ra] >= ka, lb = rootKey[rb] >= kb;
            if (la || lb) return (la && lb ? ra > rb : lb) != flip;
        }
        const uint32_t pa = ma & kMetaParent, pb = mb & kMetaParent;
        const uint32_t ca = s.comp[pa], cb = s.comp[pb];
        if (ca == cb) return (pa != pb ? s.size[pa] > s.size[pb] : a > b) != flip;
        a = ca;
        b = cb;
        flip = !flip;
    }
}

__device__ __forceinline__ uint32_t warpInclusive(uint32_t v) {
    const uint32_t lane = laneId();
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, v, o);
        if (lane >= o) v += y;
    }
    return v;
}

// ascending compare-exchange of v with lane ^ mask's
__device__ __forceinline__ unsigned long long laneExchange(unsigned long long v, uint32_t mask) {
    const unsigned long long o = __shfl_xor_sync(kFull, v, mask);
    const bool low = laneId() < (laneId() ^ mask);
    return (v < o) == low ? v : o;
}

// Ascending sort of n 64-bit values in shared memory by the group's warps: blocks of 32 in
// registers, then a bitonic network whose comparisons are all ascending (positions past the end
// need no padding), its strides below 32 in registers again.
template <int W, class Sync>
__device__ void groupSort(unsigned long long* v, uint32_t n, uint32_t wid, Sync sync) {
    constexpr uint32_t G = 32 * W;
    const uint32_t lane = laneId(), tid = wid * 32 + lane;
    for (uint32_t b = wid * 32; b < n; b += G) {
        unsigned long long x = b + lane < n ? v[b + lane] : ~0ull;
#pragma unroll
        for (uint32_t k = 2; k <= 32; k <<= 1) {
            x = laneExchange(x, k - 1);
#pragma unroll
            for (uint32_t d = k >> 2; d > 0; d >>= 1) x = laneExchange(x, d);
        }
        if (b + lane < n) v[b + lane] = x;
    }
    sync();
    auto order2 = [&](uint32_t i, uint32_t j) {
        if (j >= n) return;
        const unsigned long long x = v[i], y = v[j];
        if (y < x) {
            v[i] = y;
            v[j] = x;
        }
    };
    for (uint32_t half = 32; half < n; half <<= 1) {
        for (uint32_t t = tid; (t & ~(half - 1)) * 2 < n; t += G) {
            const uint32_t low = t & (half - 1), block = (t - low) * 2;
            order2(block + low, block + 2 * half - 1 - low);
        }
        sync();
        for (uint32_t d = half >> 1; d >= 32; d >>= 1) {
            for (uint32_t t = tid; (t & ~(d - 1)) * 2 < n; t += G) {
                const uint32_t low = t & (d - 1), block = (t - low) * 2;
                order2(block + low, block + d + low);
            }
            sync();
        }
        for (uint32_t b = wid * 32; b < n; b += G) {
            unsigned long long x = b + lane < n ? v[b + lane] : ~0ull;
#pragma unroll
            for (uint32_t d = 16; d > 0; d >>= 1) x = laneExchange(x, d);
            if (b + lane < n) v[b + lane] = x;
        }
        sync();
    }
}

// Components with equal sort keys are ordered by counting what comes before each, a comparison for every pair
// of a run. Where one root's key exceeds every key below it (the block's axis differs from the tile's, in a
// scene far from the origin) all of that root's components are one run, so a tile with a run longer than this is
// merged instead, by the kernel whose CTA has an SM (the other has no registers for it). One root of 1,783 and
// of 6,657 nodes, 128 tiles: 2,563 and 4,453 us by counting, 497 and 832 us by merging, 577 and 718
// without ties.
constexpr uint32_t kLongRun = 256;

// The components of s.sortKey into s.first in their exact order: merge passes over blocks of 1, 2, 4, ... of each
// run of equal keys, each element finding its place in the other block by bisection.
template <int W, class S>
__device__ __noinline__ void mergeRuns(S& s, const uint32_t* rootKey, uint32_t sorted) {
    uint16_t *from = s.first, *to = s.first + S::kSorted;
    // the first position whose key is not below k
    auto bound = [&](uint64_t k) {
        uint32_t lo = 0, hi = sorted;
        while (lo < hi) {
            const uint32_t mid = (lo + hi) / 2;
            if ((s.sortKey[mid] >> 32) < k) lo = mid + 1;
            else hi = mid;
        }
        return lo;
    };
    for (uint32_t e = threadIdx.x; e < sorted; e += 32 * W) from[e] = uint16_t(s.sortKey[e]);
    __syncthreads();
    for (uint32_t width = 1; width < sorted; width *= 2) {
        for (uint32_t e = threadIdx.x; e < sorted; e += 32 * W) {
            const uint64_t key = s.sortKey[e] >> 32;
            const uint32_t id = from[e], begin = bound(key), end = bound(key + 1);
            const uint32_t low = begin + ((e - begin) & ~(2 * width - 1)), mid = min(low + width, end);
            const bool left = e < mid;
            uint32_t b = left ? mid : low, t = left ? min(mid + width, end) : mid;
            const uint32_t other = b;
            while (b < t) {
                const uint32_t m = (b + t) / 2;
                if (compBefore(s, rootKey, from[m], id)) b = m + 1;
                else t = m;
            }
            to[low + (e - (left ? low : mid)) + (b - other)] = uint16_t(id);
        }
        __syncthreads();
        uint16_t* const f = from;
        from = to;
        to = f;
    }
    if (from != s.first) {
        for (uint32_t e = threadIdx.x; e < sorted; e += 32 * W) to[e] = from[e];
        __syncthreads();
    }
}

// one tile by W warps (W = 1: the calling warp alone; else the whole CTA); returns the node visits.
// overflow: the list was not made (see above); the return value is N where only the store was too small.
template <int W, uint32_t N>
__device__ uint32_t treeTile(const TileCullArgs& a, const ViewDev& V, uint32_t tile, TreeHead& h, TreeStore<N>& s,
                             bool& overflow) {
    constexpr uint32_t G = 32 * W;
    using S = TreeStore<N>;
    const uint32_t lane = laneId(), wid = W == 1 ? 0u : threadIdx.x >> 5, tid = W == 1 ? lane : threadIdx.x;
    const uint32_t q4 = lane & 28u, c = lane & 3u, below = (1u << lane) - 1u;
    auto sync = [] {
        if constexpr (W == 1) __syncwarp();
        else __syncthreads();
    };
    overflow = false;
    const uint32_t blk = tile / kTilesPerBlock;
    const uint32_t roots = V.blockSizes[blk];
    SmemFrustum& f = *reinterpret_cast<SmemFrustum*>(s.sortKey); // until the sort
    bool bad = false;
    for (uint32_t i = tid; i < roots; i += G) {
        const StackEntry e = V.blockStacks[size_t(blk) * kBlockStack + i];
        s.node[i] = e.node;
        s.comp[i] = uint16_t(i);
        s.meta[i] = i | (i << kMetaRoot) | (e.mask ? kMetaMasked : 0u);
        s.key[i] = 0;
        h.rootKey[i] = orderKey(e.tMin);
        if (isnan(e.tMin)) bad = true;
    }
    if (wid == 0) {
        buildFrustum(V.tileRays[tile], V.M, f);
        if (lane < 4) {
            h.lo[lane] = make_float4(f.tpLo[lane][0], f.tpLo[lane][1], f.tpLo[lane][2], f.w[lane]);
            h.hi[lane] = make_float4(f.tpHi[lane][0], f.tpHi[lane][1], f.tpHi[lane][2], 0.0f);
        } else if (lane < 16) {
            const uint32_t e = lane - 4, k = e % 3;
            h.edge[e] = make_float4(f.edge[e][k == 0 ? 1 : 0], f.edge[e][k == 2 ? 1 : 2], f.minF[e], f.maxF[e]);
            if (!(f.edge[e][k] == 0.0f)) bad = true; // (a direction that is not finite)
        } else if (lane < 19) {
            h.pushed[lane - 16] = 0;
        } else if (lane == 19) {
            h.total = h.sorted = 0;
            h.gen[0] = 0;
        }
    }
    const bool culled = V.hasCull && tileCulled(V.tileRays[tile], V.M, V.cull);
    sync();
    if (culled || roots == 0 || f.degenerate) {
        if (tid == 0) V.tileLists[tile] = TileList{kNoChunk, 0};
        sync();
        return 0;
    }
    // the stack is sorted from the farthest up (a caller's own block stacks may not be)
    for (uint32_t i = tid; i + 1 < roots; i += G)
        if (h.rootKey[i] < h.rootKey[i + 1]) bad = true;
    const int distIdx = f.distIdx;
    const float p0 = f.proj[0][c], p1 = f.proj[0][4 + c], p2 = f.proj[1][c], p3 = f.proj[1][4 + c],
                p4 = f.proj[2][c], p5 = f.proj[2][4 + c];
    const float* rows = reinterpret_cast<const float*>(V.nodes);

    uint32_t lo = 0, hi = roots, gens = 0, total = 0;
    for (;;) {
        uint32_t next = hi; // (W = 1) end of the next generation so far
        for (uint32_t base = lo + wid * 8; base < hi; base += 8 * W) {
            const uint32_t i = base + (lane >> 2);
            const bool act = i < hi;
            const uint32_t n = act ? s.node[i] : 0u;
            const uint32_t meta = act ? s.meta[i] : 0u;
            const float* row = rows + size_t(n) * 32;
            ChildBox b{};
            uint32_t leafMask = 0, t0 = 0, t1 = 0;
            if (act) {
                b = ChildBox{row[c], row[4 + c], row[8 + c], row[12 + c], row[16 + c], row[20 + c]};
                leafMask = __float_as_uint(row[24]);
                t0 = __float_as_uint(row[25 + c]);
                t1 = __float_as_uint(row[26 + c]);
            }
            // testBVHNodeChildren
            bool pass = act & (b.xM >= p0) & (b.xN >= p1) & (b.yM >= p2) & (b.yN >= p3) & (b.zM >= p4) & (b.zN >= p5);
#pragma unroll
            for (int p = 0; p < 4; p++) {
                const float4 l = h.lo[p], u = h.hi[p];
                const float dl = fmaf(l.x, b.xM, fmaf(l.y, b.yM, l.z * b.zM));
                const float du = fmaf(u.x, b.xN, fmaf(u.y, b.yN, u.z * b.zN));
                pass = pass & ((dl + du) <= l.w);
            }
            // testBVHNodeChildrenRefine, for every child of a node with a passing leaf
            const bool leafy = ((__ballot_sync(kFull, pass) >> q4) & 15u & leafMask) != 0;
            const bool refine = pass & leafy;
            if (__any_sync(kFull, refine)) {
                bool reject = false;
#pragma unroll
                for (int e = 0; e < 12; e += 3) {
                    const float4 ex = h.edge[e], ey = h.edge[e + 1], ez = h.edge[e + 2];
                    reject = reject | edgeReject2(b.yM, b.yN, b.zM, b.zN, ex) | edgeReject2(b.xM, b.xN, b.zM, b.zN, ey) |
                             edgeReject2(b.xM, b.xN, b.yM, b.yN, ez);
                }
                pass = pass & !(refine & reject);
                // a zero component's product is zero (so edgeReject2 can leave it out) only for finite bounds
                if (refine && !(fabsf(((b.xM + b.xN) + (b.yM + b.yN)) + (b.zM + b.zN)) <= FLT_MAX)) bad = true;
            }
            const bool leaf = (leafMask >> c) & 1u;
            uint32_t len = 0;
            if (pass & leaf) {
                if (t1 <= t0) {
                    atomicOr(&a.counters[1], kStatusBadLeaf);
                } else {
                    len = t1 - t0;
                    if (len > kMaxLeafRange) bad = true, len = 1;
                }
            }
            const uint32_t leafBits = (__ballot_sync(kFull, len != 0) >> q4) & 15u;
            total += len;
            // the internal children that pass are the next generation's nodes
            const bool push = pass & !leaf & !(meta & kMetaMasked);
            const uint32_t pb = __ballot_sync(kFull, push);
            const uint32_t m = __popc((pb >> q4) & 15u);
            uint32_t at = next;
            if constexpr (W == 1) {
                next += __popc(pb);
            } else if (pb) {
                if (lane == 0) at = hi + atomicAdd(&h.pushed[gens % 3u], uint32_t(__popc(pb)));
                at = __shfl_sync(kFull, at, 0);
            }
            const uint32_t pos = at + __popc(pb & below);
            const uint32_t comp = act ? s.comp[i] : 0u;
            if (push & (pos < N)) {
                uint32_t cid = comp;
                if (m > 1) {
                    const float v = distIdx < 2 ? (distIdx == 0 ? b.xM : b.xN)
                                                : (distIdx < 4 ? (distIdx == 2 ? b.yM : b.yN) : (distIdx == 4 ? b.zM : b.zN));
                    const uint32_t key = orderKey(-v), parentKey = s.key[comp];
                    if (key < parentKey || isnan(v)) bad = true;
                    if (key != parentKey) {
                        cid = pos;
                        s.key[pos] = key;
                    }
                }
                s.node[pos] = n + t1;
                s.comp[pos] = uint16_t(cid);
                s.meta[pos] = i | (s.meta[comp] & (63u << kMetaRoot));
                asm volatile("prefetch.global.L1 [%0];" ::"l"(rows + size_t(n + t1) * 32));
            }
            __syncwarp();
            if (act & (c == 0)) {
                s.first[i] = uint16_t(at + __popc(pb & below));
                atomicOr(&s.meta[i], (leafBits << kMetaSlots) | (m << kMetaChildren));
                if (leafBits) atomicOr(&s.meta[comp], kMetaLeafy);
            }
        }
        if constexpr (W == 1) {
            if (__any_sync(kFull, bad)) next = kPushedBad;
            __syncwarp();
        } else {
            if (bad) atomicAdd(&h.pushed[gens % 3u], kPushedBad);
            __syncthreads();
            next = hi + h.pushed[gens % 3u];
            if (tid == 0) h.pushed[(gens + 2u) % 3u] = 0; // (read before the last barrier, used after the next)
        }
        ++gens;
        if (tid == 0) h.gen[gens] = uint16_t(hi);
        if (next > N || (gens >= kMaxGens && next != hi)) {
            overflow = true;
            sync();
            return next > N && next < kPushedBad ? N : min(hi, N - 1);
        }
        if (next == hi) break;
        lo = hi;
        hi = next;
    }
    const uint32_t visits = hi;
    total = __reduce_add_sync(kFull, total);
    if constexpr (W > 1) {
        if (lane == 0 && total) atomicAdd(&h.total, total);
        __syncthreads();
        total = h.total;
    }
    if (total == 0) {
        if (tid == 0) V.tileLists[tile] = TileList{kNoChunk, 0};
        sync();
        return visits;
    }
    // depth-first offsets inside the components: subtree sizes upwards, offsets downwards
    for (uint32_t g = gens; g-- > 0;) {
        for (uint32_t i = h.gen[g] + tid; i < h.gen[g + 1]; i += G) {
            const uint32_t m = (s.meta[i] >> kMetaChildren) & 7u, fc = s.first[i], own = s.comp[i];
            uint32_t z = 1;
#pragma unroll
            for (uint32_t k = 0; k < 4; k++)
                if (k < m && s.comp[fc + k] == own) z += s.size[fc + k];
            s.size[i] = uint16_t(z);
            if (g == 0) s.compSize[i] = uint16_t(z);
        }
        sync();
    }
    for (uint32_t i = tid; i < roots; i += G) s.size[i] = 0;
    sync();
    for (uint32_t g = 0; g + 1 < gens; g++) {
        for (uint32_t i = h.gen[g] + tid; i < h.gen[g + 1]; i += G) {
            const uint32_t m = (s.meta[i] >> kMetaChildren) & 7u, fc = s.first[i], own = s.comp[i];
            uint32_t off = s.size[i] + 1u, z[4], cid[4];
#pragma unroll
            for (uint32_t k = 0; k < 4; k++) {
                z[k] = k < m ? s.size[fc + k] : 0u;
                cid[k] = k < m ? s.comp[fc + k] : 0u;
            }
#pragma unroll
            for (int k = 3; k >= 0; k--) {
                if (uint32_t(k) >= m) continue;
                if (cid[k] == own) {
                    s.size[fc + k] = uint16_t(off);
                    off += z[k];
                } else {
                    s.compSize[cid[k]] = uint16_t(z[k]);
                    s.size[fc + k] = 0;
                }
            }
        }
        sync();
    }
    // the components with passing leaves, by largest key on the path
    uint32_t sorted = 0;
    for (uint32_t b = wid * 32; b < visits; b += G) {
        const uint32_t i = b + lane;
        const uint32_t meta = i < visits && s.comp[i] == i ? s.meta[i] : 0u;
        const uint32_t on = __ballot_sync(kFull, meta & kMetaLeafy);
        uint32_t pos = sorted;
        if constexpr (W == 1) {
            sorted += __popc(on);
        } else if (on) {
            if (lane == 0) pos = atomicAdd(&h.sorted, uint32_t(__popc(on)));
            pos = __shfl_sync(kFull, pos, 0);
        }
        pos += __popc(on & below);
        if ((meta & kMetaLeafy) && pos < S::kSorted)
            s.sortKey[pos] = (uint64_t(max(h.rootKey[(meta >> kMetaRoot) & 63u], s.key[i])) << 32) | i;
    }
    sync();
    if constexpr (W > 1) sorted = h.sorted;
    if (sorted > S::kSorted) {
        overflow = true;
        sync();
        return N;
    }
    groupSort<W>(s.sortKey, sorted, wid, sync);
    // runs of equal keys in their exact order
    uint16_t* ordered = s.first;
    bool longRun = false; // (a warp's are short)
    for (uint32_t e = tid; e < sorted; e += G) {
        const unsigned long long v = s.sortKey[e];
        const uint32_t key = uint32_t(v >> 32), id = uint32_t(v);
        uint32_t pos = e;
        if (W > 1 && ((e >= kLongRun && uint32_t(s.sortKey[e - kLongRun] >> 32) == key) ||
                      (e + kLongRun < sorted && uint32_t(s.sortKey[e + kLongRun] >> 32) == key))) {
            longRun = true;
            continue;
        }
        for (uint32_t j = e; j-- > 0;) {
            const unsigned long long o = s.sortKey[j];
            if (uint32_t(o >> 32) != key) break;
            if (!compBefore(s, h.rootKey, uint32_t(o), id)) pos--;
        }
        for (uint32_t j = e + 1; j < sorted; j++) {
            const unsigned long long o = s.sortKey[j];
            if (uint32_t(o >> 32) != key) break;
            if (compBefore(s, h.rootKey, uint32_t(o), id)) pos++;
        }
        ordered[pos] = uint16_t(id);
    }
    if constexpr (W == 1) {
        __syncwarp();
    } else if (__syncthreads_or(longRun)) {
        if constexpr (W < int(kHugeWarps)) { // (left to the kernel that merges)
            overflow = true;
            return visits;
        } else {
            mergeRuns<W>(s, h.rootKey, sorted);
        }
    }
    // the list's chunks, consecutive in the pool: taken once nothing can send the tile to another cull any
    // more, so that a pool that holds the lists is always enough
    const uint32_t chunks = (total + kChunk - 1) / kChunk;
    uint32_t chunk0 = 0;
    if (tid == 0) {
        chunk0 = atomicAdd(&a.counters[0], chunks);
        if (W > 1) h.first = chunk0;
    }
    __syncwarp();
    // the components' first positions
    uint32_t placed = 0;
    for (uint32_t b = 0; b < sorted; b += G) {
        const uint32_t j = b + tid;
        const uint32_t cid = j < sorted ? ordered[j] : 0u;
        const uint32_t z = j < sorted ? s.compSize[cid] : 0u;
        const uint32_t inc = warpInclusive(z);
        uint32_t start = placed;
        if constexpr (W > 1) {
            if (lane == 31) h.warpSum[wid] = inc;
            __syncthreads();
            uint32_t all = 0;
#pragma unroll
            for (uint32_t w = 0; w < uint32_t(W); w++) {
                if (w < wid) start += h.warpSum[w];
                all += h.warpSum[w];
            }
            placed += all;
            __syncthreads();
        } else {
            placed += __shfl_sync(kFull, inc, 31);
        }
        if (j < sorted) s.compSize[cid] = uint16_t(start + inc - z);
    }
    sync();
    uint16_t* at = s.first;
    for (uint32_t i = tid; i < visits; i += G) {
        const uint32_t cid = s.comp[i];
        if (s.meta[cid] & kMetaLeafy) at[s.compSize[cid] + s.size[i]] = uint16_t(i);
    }
    if constexpr (W == 1) chunk0 = __shfl_sync(kFull, chunk0, 0);
    else chunk0 = h.first;
    sync();
    if (chunk0 >= a.poolChunks || chunks > a.poolChunks - chunk0) {
        if (tid == 0) {
            atomicOr(&a.counters[1], kStatusPoolOverflow);
            V.tileLists[tile] = TileList{kNoChunk, 0};
        }
        sync();
        return visits;
    }
    for (uint32_t k = tid; k < chunks; k += G) a.chunkNext[chunk0 + k] = k + 1 < chunks ? chunk0 + k + 1 : kNoChunk;
    // the list: groups of 32 nodes in order, a lane per node; a group's entries are gathered in shared
    // memory (the sort's) and written out together
    uint32_t* out = a.pool + size_t(chunk0) * kChunk;
    constexpr uint32_t kStageEntries = 2 * S::kSorted / W;
    uint32_t* stage = reinterpret_cast<uint32_t*>(s.sortKey) + wid * kStageEntries;
    uint32_t* groupAt = s.key; // (its last use was the runs' order)
    const uint32_t groups = (placed + 31) / 32;
    struct Leaves {
        uint32_t t[5], bits, count;
    };
    auto leavesOf = [&](uint32_t g) {
        Leaves r;
        r.bits = r.count = 0;
        const uint32_t j = g * 32 + lane;
        const uint32_t i = j < placed ? at[j] : 0u;
        if (j < placed) r.bits = (s.meta[i] >> kMetaSlots) & 15u;
        if (r.bits) {
            const uint4* w = reinterpret_cast<const uint4*>(rows + size_t(s.node[i]) * 32 + 24);
            const uint4 w0 = __ldg(w), w1 = __ldg(w + 1);
            r.t[0] = w0.y; r.t[1] = w0.z; r.t[2] = w0.w; r.t[3] = w1.x; r.t[4] = w1.y;
#pragma unroll
            for (int k = 0; k < 4; k++)
                if ((r.bits >> k) & 1u) r.count += r.t[k + 1] - r.t[k];
        }
        return r;
    };
    if constexpr (W > 1) {
        for (uint32_t g = wid; g < groups; g += W) {
            const uint32_t n = __reduce_add_sync(kFull, leavesOf(g).count);
            if (lane == 0) groupAt[g] = n;
        }
        __syncthreads();
        if (wid == 0) {
            uint32_t run = 0;
            for (uint32_t b = 0; b < groups; b += 32) {
                const uint32_t n = b + lane < groups ? groupAt[b + lane] : 0u;
                const uint32_t inc = warpInclusive(n);
                if (b + lane < groups) groupAt[b + lane] = run + inc - n;
                run += __shfl_sync(kFull, inc, 31);
            }
        }
        __syncthreads();
    }
    uint32_t base = 0;
    for (uint32_t g = wid; g < groups; g += W) {
        const Leaves r = leavesOf(g);
        const uint32_t inc = warpInclusive(r.count);
        const uint32_t n = __shfl_sync(kFull, inc, 31);
        if constexpr (W > 1) base = groupAt[g];
        const bool staged = n <= kStageEntries;
        uint32_t* dst = (staged ? stage : out + base) + (inc - r.count);
        if (r.bits) {
#pragma unroll
            for (int k = 0; k < 4; k++)
                if ((r.bits >> k) & 1u)
                    for (uint32_t t = r.t[k]; t < r.t[k + 1]; t++) *dst++ = t;
        }
        if (staged) {
            __syncwarp();
            for (uint32_t e = lane; e < n; e += 32) out[base + e] = stage[e];
            __syncwarp();
        }
        base += n;
    }
    if (tid == 0) V.tileLists[tile] = TileList{chunk0, total};
    return visits;
}

// Persistent CTAs. The tiles that were large in the last frame (a.counts[0] tiles at the front of the
// class's order, of which the first a.counts[1] are culled by tileTreeHugeKernel) are culled by a whole
// CTA each, then every warp takes small ones; a small one that outgrows its warp's store is kept in a
// list of its CTA (linked through the tiles' unwritten TileLists) and culled by the whole CTA once its
// warps are done. Tiles that outgrow the CTA's store go to the retry list. Non-persistent: a CTA takes
// one large tile, or one small one per warp.
__global__ void __launch_bounds__(kTreeWarps * 32, 4) tileTreeKernel(TileCullArgs a) {
    extern __shared__ __align__(16) unsigned char treeRaw[];
    TreeSmem& sm = *reinterpret_cast<TreeSmem*>(treeRaw);
    // (a following launch with programmatic serialization may start once every CTA of this grid runs)
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const uint32_t warp = threadIdx.x >> 5, lane = laneId();
    const uint32_t huge = a.huge(), big = a.big();
    auto viewOf = [&](uint32_t gt) -> const ViewDev& { return viewOfBlock(a.views, a.blockView, a.viewCount, gt / kTilesPerBlock); };
    auto ctaTile = [&](uint32_t gt) {
        const ViewDev& V = viewOf(gt);
        const uint32_t tile = gt - V.tileStart;
        bool overflow;
        const uint32_t visits = treeTile<kTreeWarps>(a, V, tile, sm.head[0], sm.cta, overflow);
        if (threadIdx.x == 0) {
            V.tileCost[tile] = visits;
            if (overflow) {
                V.tileLists[tile] = TileList{kNoChunk, 0};
                a.retry[a.first + atomicAdd(a.retryCount, 1u)] = gt;
            }
        }
        publishTile<kTreeWarps>(a, gt, overflow);
    };
    if (threadIdx.x == 0) sm.spill = kNoChunk;
    bool tookBig = false;
    for (;;) {
        if (threadIdx.x == 0) sm.item = huge + atomicAdd(a.bigQueue, 1u);
        __syncthreads();
        const uint32_t w = sm.item;
        __syncthreads();
        if (w >= big) break;
        tookBig = true;
        ctaTile(a.order ? a.order[a.first + w] : a.first + w);
        if (!a.persistent) break;
    }
    while (a.persistent || !tookBig) {
        uint32_t w = 0;
        if (lane == 0) w = atomicAdd(a.queue, 1u);
        w = big + __shfl_sync(kFull, w, 0);
        if (w >= a.count) break;
        const uint32_t gt = a.order ? a.order[a.first + w] : a.first + w;
        const ViewDev& V = viewOf(gt);
        const uint32_t tile = gt - V.tileStart;
        bool overflow;
        const uint32_t visits = treeTile<1>(a, V, tile, sm.head[warp], sm.warp[warp], overflow);
        if (overflow) {
            if (lane == 0) V.tileLists[tile].first = atomicExch(&sm.spill, gt);
        } else {
            if (lane == 0) V.tileCost[tile] = visits;
            publishTile<1>(a, gt, false);
        }
        __syncwarp();
        if (!a.persistent) break;
    }
    __syncthreads();
    for (uint32_t gt = sm.spill; gt != kNoChunk;) {
        const ViewDev& V = viewOf(gt);
        const uint32_t next = *reinterpret_cast<volatile uint32_t*>(&V.tileLists[gt - V.tileStart].first);
        __syncthreads();
        ctaTile(gt);
        __syncthreads();
        gt = next;
    }
    // this grid ends after the one that it started beside (tileTreeHugeKernel), so that a later launch
    // finds both lists' tiles complete
    if (blockIdx.x == 0 && threadIdx.x == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
}

// The tiles that a whole SM's shared memory is for. LIST = false: the class's tiles that were this
// large in the last frame, before its other tiles (a tile that outgrows the store, or cannot be
// culled breadth first, goes to the retry list). LIST = true: the retry list; what no store can
// take, and every tile when tree is 0, is culled by one warp with the sequential traversal and the
// reference's TileFrame capacity (4096 entries, 48 KiB).
// A tile above kHugeNodes (a giant) has its store in global memory, of which a frame of one rate class has
// kGiantSlots once a frame has shown such tiles: where last frame's visits say so at once, else, or with no slot
// left, in the retry pass, marked in the list (kRetryGiant) and taken by its first kGiantSlots CTAs. Node by node
// such a tile holds its warp, and the shade behind it, for 10 to 30 ms. Frames with the sequential kernel for them and
// so: 1M triangles N = 8 320 x 240 17.2 and 4.6 ms, 160 x 120 29.8 and 6.7; 300k triangles from far above 1920 x 1080
// N = 2 22.5 and 4.7.
template <bool LIST>
__global__ void __launch_bounds__(kHugeWarps * 32, 1) tileTreeHugeKernel(TileCullArgs a, uint32_t tree) {
    extern __shared__ __align__(16) unsigned char treeRaw[];
    HugeSmem& sm = *reinterpret_cast<HugeSmem*>(treeRaw);
    // (the retry pass: the cull, where the launch was scheduled before its end)
    if (LIST) asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    using Giant = TreeStore<kGiantNodes>;
    Giant* const giants = static_cast<Giant*>(a.giants);
    const uint32_t count = LIST ? *reinterpret_cast<volatile uint32_t*>(a.retryCount) : a.huge();
    auto next = [&](uint32_t* queue) { // the queue's next number, for the CTA
        if (threadIdx.x == 0) sm.item = atomicAdd(queue, 1u);
        __syncthreads();
        const uint32_t n = sm.item;
        __syncthreads();
        return n;
    };
    auto viewOf = [&](uint32_t gt) -> const ViewDev& { return viewOfBlock(a.views, a.blockView, a.viewCount, gt / kTilesPerBlock); };
    auto giantTile = [&](const ViewDev& V, uint32_t tile, uint32_t slot, bool& overflow) {
        const uint32_t visits = treeTile<kHugeWarps>(a, V, tile, sm.head, giants[slot], overflow);
        __syncthreads();
        return visits;
    };
    // (LIST) what no store took
    auto sequential = [&](const ViewDev& V, uint32_t tile, uint32_t visits) {
        if (threadIdx.x < 32) {
            bool overflow;
            visits = cullTile(a, V, tile, sm.seq, overflow);
            if (overflow && threadIdx.x == 0) atomicOr(&a.counters[1], kStatusStackOverflow);
        }
        return visits;
    };
    uint32_t slot = ~0u; // (LIST = false) the CTA's store in global memory
    for (uint32_t w = blockIdx.x; w < count; w += gridDim.x) {
        const uint32_t entry = LIST ? a.retry[a.first + w] : a.order[a.first + w], gt = entry & ~kRetryGiant;
        if (LIST && entry != gt) continue; // (below)
        const ViewDev& V = viewOf(gt);
        const uint32_t tile = gt - V.tileStart;
        const uint32_t last = V.tileCost[tile]; // (LIST = false: last frame's visits)
        bool overflow = true, giant = !LIST && giants && last > kHugeNodes;
        uint32_t visits = last;
        if (giant) {
            if (slot == ~0u) slot = next(a.giantSlots);
            if (slot < kGiantSlots) {
                visits = giantTile(V, tile, slot, overflow);
                giant = false;
            }
        } else if (tree) {
            visits = treeTile<kHugeWarps>(a, V, tile, sm.head, sm.cta, overflow);
            giant = overflow && visits == kHugeNodes;
            __syncthreads();
            if (LIST && giant && threadIdx.x == 0) atomicAdd(&a.counters[kGiantWord], 1u);
            if (LIST && giant && giants && blockIdx.x < kGiantSlots) visits = giantTile(V, tile, blockIdx.x, overflow);
        }
        if (LIST && overflow) visits = sequential(V, tile, visits);
        if (threadIdx.x == 0) {
            V.tileCost[tile] = visits;
            if (!LIST && overflow) {
                V.tileLists[tile] = TileList{kNoChunk, 0};
                a.retry[a.first + atomicAdd(a.retryCount, 1u)] = gt | (giant && giants ? kRetryGiant : 0u);
            }
        }
        if (!LIST) publishTile<kHugeWarps>(a, gt, overflow);
        __syncthreads();
    }
    if (!LIST || !giants || blockIdx.x >= kGiantSlots) return;
    for (uint32_t w = next(a.giantQueue); w < count; w = next(a.giantQueue)) {
        const uint32_t entry = a.retry[a.first + w], gt = entry & ~kRetryGiant;
        if (entry == gt) continue;
        const ViewDev& V = viewOf(gt);
        const uint32_t tile = gt - V.tileStart;
        bool overflow;
        uint32_t visits = giantTile(V, tile, blockIdx.x, overflow);
        if (overflow) visits = sequential(V, tile, visits);
        if (threadIdx.x == 0) V.tileCost[tile] = visits;
        __syncthreads();
    }
}

// Orders the global tiles by (rate class ascending, cost descending), cost in quarter octaves
// of last frame's visit counts, and counts each class's large tiles (their buckets lie at the front
// of the class). One block; positions within a bucket are in arrival order.
constexpr uint32_t kCostBuckets = 132, kOrderBuckets = kRateClasses * kCostBuckets;
constexpr uint32_t kOrderPerThread = (kOrderBuckets + 1023) / 1024;
__host__ __device__ constexpr uint32_t costBucket(uint32_t c, uint32_t log2) { return kCostBuckets - 1 - (log2 * 4 + (((c + 1) << (31 - log2)) >> 29 & 3u)); }
// A tile of at least kBigCost visits is culled by a whole CTA and one of at least kHugeCost by a CTA
// with an SM's shared memory: bucket bounds that leave a warp's store (kWarpNodes) a third and a
// CTA's (kCtaNodes) an eighth of headroom for a view that moves between frames (a tile of which more than
// half of the store's nodes are list-bearing components outgrows the store earlier; a huge tile holds a
// whole SM: starting them at 1,536 visits took 6.0 ms instead of 2.8 for the cull of a foveated
// frame with a thousand of them).
constexpr uint32_t kBigCost = 191, kHugeCost = 1791;
constexpr uint32_t kBigBuckets = costBucket(kBigCost, 7) + 1, kHugeBuckets = costBucket(kHugeCost, 10) + 1;
// A CTA has eight warps for a tile's generations, and kFewTiles of them (four on each of 148 SMs) are
// resident at once: where no more tiles than that reach 47 or 95 visits, those get a CTA as well. Cull
// of a view of 2,400 tiles alone: 85 -> 53 us; frames 233 against 240 us and 360 against 371, thin lens
// 457 against 483; nothing where more tiles reach 95. With two an SM (296) the frames were unchanged.
constexpr uint32_t kFewTiles = 592, kFewBuckets47 = costBucket(47, 5) + 1, kFewBuckets95 = costBucket(95, 6) + 1;
__global__ void __launch_bounds__(1024) tileOrderKernel(FrameDev fr) {
    __shared__ uint32_t hist[kOrderPerThread * 1024];
    __shared__ uint32_t warpSum[32];
    const uint32_t tid = threadIdx.x, lane = laneId();
    for (uint32_t b = tid; b < kOrderPerThread * 1024; b += 1024) hist[b] = 0;
    __syncthreads();
    auto bucket = [&](uint32_t t) {
        const ViewDev& V = viewOfBlock(fr.views, fr.blockView, fr.viewCount, t / kTilesPerBlock);
        const uint32_t c = min(V.tileCost[t - V.tileStart], 0x7ffffffeu);
        return V.rateIdx * kCostBuckets + costBucket(c, 31u - __clz(c + 1u));
    };
    for (uint32_t t = tid; t < fr.tiles; t += 1024) atomicAdd(&hist[bucket(t)], 1u);
    __syncthreads();
    uint32_t mine[kOrderPerThread], sum = 0;
#pragma unroll
    for (uint32_t k = 0; k < kOrderPerThread; k++) {
        mine[k] = sum;
        sum += hist[tid * kOrderPerThread + k];
    }
    uint32_t inc = sum;
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, inc, o);
        if (lane >= o) inc += y;
    }
    if (lane == 31) warpSum[tid >> 5] = inc;
    __syncthreads();
    if (tid < 32) {
        const uint32_t n = warpSum[lane];
        uint32_t w = n;
#pragma unroll
        for (uint32_t o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(kFull, w, o);
            if (lane >= o) w += y;
        }
        warpSum[lane] = w - n;
    }
    __syncthreads();
    const uint32_t base = warpSum[tid >> 5] + inc - sum;
#pragma unroll
    for (uint32_t k = 0; k < kOrderPerThread; k++) hist[tid * kOrderPerThread + k] = base + mine[k];
    __syncthreads();
    // (the exclusive prefix before the scatter moves it)
    if (fr.bigCountOut && tid < kBigWords * kRateClasses) {
        const uint32_t* h = hist + tid / kBigWords * kCostBuckets;
        const uint32_t word = tid % kBigWords;
        uint32_t n = h[word == 1 ? kHugeBuckets : kBigBuckets] - h[0];
        if (word == 0) {
            if (h[kFewBuckets95] - h[0] <= kFewTiles) n = h[kFewBuckets95] - h[0];
            if (h[kFewBuckets47] - h[0] <= kFewTiles) n = h[kFewBuckets47] - h[0];
        }
        if (word == 2 && (n > kSplitTiles || h[kFewBuckets47] - h[0] > kFewTiles)) n = 0;
        fr.bigCountOut[tid] = n;
    }
    __syncthreads();
    for (uint32_t t = tid; t < fr.tiles; t += 1024) fr.order[atomicAdd(&hist[bucket(t)], 1u)] = t;
}

__global__ void writeViewKernel(ViewDev v, ViewDev* dst) { *dst = v; }

// The reference runs its intersect and resolve kernels over the compacted list of occupied tiles
// (tileIndexRemapOccupied, libraries/hvvr/raycaster/traversal.cpp:213-330) and indexes the lens
// table by that CTA index; this is each tile's rank among the view's non-empty tiles.
__global__ void __launch_bounds__(1024) occupiedRankKernel(FrameDev fr) {
    const ViewDev& V = fr.views[blockIdx.x];
    if (!(V.lensRadius > 0.0f)) return;
    __shared__ uint32_t warpSums[32];
    __shared__ uint32_t carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    const uint32_t lane = laneId(), warp = threadIdx.x >> 5;
    const uint32_t tiles = (blockIdx.x + 1 < fr.viewCount ? fr.views[blockIdx.x + 1].tileStart : fr.tiles) - V.tileStart;
    for (uint32_t base = 0; base < tiles; base += 1024) {
        const uint32_t t = base + threadIdx.x;
        const uint32_t occ = (t < tiles && V.tileLists[t].count > 0) ? 1u : 0u;
        const uint32_t bal = __ballot_sync(kFull, occ);
        if (lane == 0) warpSums[warp] = __popc(bal);
        __syncthreads();
        uint32_t before = carry;
        for (uint32_t w = 0; w < warp; w++) before += warpSums[w];
        if (t < tiles) V.occRank[t] = before + __popc(bal & ((1u << lane) - 1u));
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t sum = 0;
            for (uint32_t w = 0; w < 32; w++) sum += warpSums[w];
            carry += sum;
        }
        __syncthreads();
    }
}

struct DeviceLimits {
    int sms = 0;
    int ctasPerSm[9] = {};  // indexed by warps per CTA
    bool treeReady = false;
};

// per-device launch limits, filled on first use; host threads rendering on different streams
// may get here together, so the first use of a device is serialised
std::mutex gLimitsMutex;

DeviceLimits& limits() {
    static DeviceLimits perDevice[64];
    int dev = 0;
    cudaGetDevice(&dev);
    DeviceLimits& d = perDevice[dev < 0 || dev >= 64 ? 0 : dev];
    std::lock_guard<std::mutex> lock(gLimitsMutex);
    if (!d.sms) {
        int sms = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        d.sms = sms < 1 ? 1 : sms;
    }
    return d;
}

template <int W>
cudaError_t launchTileCullW(const TileCullArgs& a, uint32_t count, uint32_t capPerSm, cudaStream_t st) {
    if (!a.persistent) {
        tileCullKernel<W><<<(count + W - 1) / W, W * 32, 0, st>>>(a);
        return cudaGetLastError();
    }
    DeviceLimits& d = limits();
    {
        std::lock_guard<std::mutex> lock(gLimitsMutex);
        if (!d.ctasPerSm[W]) {
            int occ = 0;
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, tileCullKernel<W>, W * 32, 0);
            d.ctasPerSm[W] = occ < 1 ? 1 : occ;
        }
    }
    const uint32_t needed = (count + W - 1) / W;
    const uint32_t perSm = capPerSm ? std::min<uint32_t>(capPerSm, uint32_t(d.ctasPerSm[W])) : uint32_t(d.ctasPerSm[W]);
    const uint32_t grid = std::min<uint32_t>(needed, uint32_t(d.sms) * perSm);
    tileCullKernel<W><<<grid, W * 32, 0, st>>>(a);
    return cudaGetLastError();
}

// shared-memory sizes above the default, set once per device
cudaError_t treeReady(DeviceLimits& d) {
    std::lock_guard<std::mutex> lock(gLimitsMutex);
    if (d.treeReady) return cudaSuccess;
    const cudaFuncAttribute at = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaError_t e = cudaFuncSetAttribute(tileTreeKernel, at, int(sizeof(TreeSmem)));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(tileTreeHugeKernel<false>, at, int(sizeof(HugeSmem)));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(tileTreeHugeKernel<true>, at, int(sizeof(HugeSmem)));
    d.treeReady = e == cudaSuccess;
    return e;
}

cudaError_t launchTileTree(const TileCullArgs& a, uint32_t capPerSm, cudaStream_t st) {
    DeviceLimits& d = limits();
    cudaError_t e = treeReady(d);
    if (e != cudaSuccess) return e;
    // (how many tiles are large is known on the device only, so a CTA per tile, up to what is resident)
    const uint32_t resident = uint32_t(d.sms) * (capPerSm ? std::min(capPerSm, 4u) : 4u);
    const uint32_t grid = a.persistent ? std::min(a.count, resident) : a.count;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kTreeWarps * 32);
    cfg.dynamicSmemBytes = sizeof(TreeSmem);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    if (a.counts && !a.noHuge) {
        tileTreeHugeKernel<false><<<std::min<uint32_t>(a.count, d.sms), kHugeWarps * 32, sizeof(HugeSmem), st>>>(a, 1u);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        // the other tiles' cull starts beside it, once its CTAs run
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }
    return cudaLaunchKernelEx(&cfg, tileTreeKernel, a);
}

// the retry pass: it reads the retry count on the device and exits at once when the list is empty. early: the
// launch before it in the stream is the cull, and this one may be scheduled before that ends
cudaError_t launchTileCullRetry(const TileCullArgs& a, bool tree, bool early, cudaStream_t st) {
    DeviceLimits& d = limits();
    const cudaError_t e = treeReady(d);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(std::min<uint32_t>(a.count, d.sms));
    cfg.blockDim = dim3(kHugeWarps * 32);
    cfg.dynamicSmemBytes = sizeof(HugeSmem);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = early ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, tileTreeHugeKernel<true>, a, tree ? 1u : 0u);
}

} // namespace

size_t giantStoreBytes() { return kGiantSlots * sizeof(TreeStore<kGiantNodes>); }

cudaError_t launchBlockCull(const FrameDev& fr, cudaStream_t st) {
    if (fr.blocks == 0) return cudaSuccess;
    blockCullKernel<<<fr.blocks + kPrefetchCtas, kBlockWarps * 32, 0, st>>>(fr);
    return cudaGetLastError();
}

cudaError_t launchTileOrder(const FrameDev& fr, cudaStream_t st) {
    if (fr.tiles == 0) return cudaSuccess;
    tileOrderKernel<<<1, 1024, 0, st>>>(fr);
    return cudaGetLastError();
}

cudaError_t launchTileCullMain(const FrameDev& fr, const uint32_t* order, uint32_t first, uint32_t count,
                               uint32_t* queues, uint32_t warps, uint32_t stackLimit, uint32_t* ready,
                               uint32_t* readyTail, cudaStream_t st) {
    if (count == 0) return cudaSuccess;
    if (stackLimit == 0) {
        const TileCullArgs t{fr.views, fr.blockView, fr.viewCount, fr.pool, fr.chunkNext, fr.poolChunks, fr.counters,
                             order, first, count, queues, fr.retry, queues + 1, kTileStack, ready, readyTail,
                             fr.cullPersistent ? 1u : 0u, order ? fr.bigCount : nullptr, fr.noHuge, queues + 2,
                             fr.giants, queues + 3, queues + 4};
        return launchTileTree(t, fr.cullCtasPerSm, st);
    }
    if (stackLimit > kTileStack) stackLimit = kTileStack;
    if (stackLimit < 8) return cudaErrorInvalidValue;
    const TileCullArgs a{fr.views, fr.blockView, fr.viewCount, fr.pool, fr.chunkNext, fr.poolChunks, fr.counters,
                         order, first, count, queues, fr.retry, queues + 1, stackLimit, ready, readyTail,
                         fr.cullPersistent ? 1u : 0u, nullptr, 0u, nullptr, nullptr, nullptr, nullptr};
    switch (warps) {
    case 1: return launchTileCullW<1>(a, count, fr.cullCtasPerSm, st);
    case 2: return launchTileCullW<2>(a, count, fr.cullCtasPerSm, st);
    case 4: return launchTileCullW<4>(a, count, fr.cullCtasPerSm, st);
    case 8: return launchTileCullW<8>(a, count, fr.cullCtasPerSm, st);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t launchTileCullRetryPass(const FrameDev& fr, const uint32_t* order, uint32_t first, uint32_t count,
                                    uint32_t* queues, uint32_t stackLimit, bool early, cudaStream_t st) {
    if (count == 0) return cudaSuccess;
    const TileCullArgs a{fr.views, fr.blockView, fr.viewCount, fr.pool, fr.chunkNext, fr.poolChunks, fr.counters,
                         order, first, count, queues, fr.retry, queues + 1, kTileStack, nullptr, nullptr, 1u,
                         nullptr, 0u, nullptr, fr.giants, queues + 3, queues + 4};
    return launchTileCullRetry(a, stackLimit == 0, early, st);
}

cudaError_t launchTileCull(const FrameDev& fr, const uint32_t* order, uint32_t first, uint32_t count,
                           uint32_t* queues, uint32_t warps, uint32_t stackLimit, bool early, cudaStream_t st) {
    const cudaError_t e = launchTileCullMain(fr, order, first, count, queues, warps, stackLimit, nullptr, nullptr, st);
    if (e != cudaSuccess) return e;
    return launchTileCullRetryPass(fr, order, first, count, queues, stackLimit, early && stackLimit == 0, st);
}

cudaError_t launchOccupiedRank(const FrameDev& fr, cudaStream_t st) {
    if (fr.viewCount == 0) return cudaSuccess;
    occupiedRankKernel<<<fr.viewCount, 1024, 0, st>>>(fr);
    return cudaGetLastError();
}

cudaError_t launchWriteView(const ViewDev& v, ViewDev* dst, cudaStream_t st) {
    writeViewKernel<<<1, 1, 0, st>>>(v, dst);
    return cudaGetLastError();
}

} // namespace hvb

#ifdef HVVR_VISIT_CLOCKS
// profiling build only: per global tile [0, tiles), kVcPhases phase cycle sums then the visit count
extern "C" int hvvr_dbg_visit_clocks(unsigned long long* out, uint32_t tiles) {
    if (!out || tiles > hvb::kVisitClockTiles) return HVVR_ERR_INVALID;
    return cudaMemcpyFromSymbol(out, hvb::gVisitClocks, size_t(tiles) * sizeof(hvb::gVisitClocks[0])) == cudaSuccess
               ? HVVR_OK
               : HVVR_ERR_CUDA;
}
#endif
