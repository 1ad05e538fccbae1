// GPU BVH builder (see build.cuh).
//
// Binary phase: top-down binned SAH (32 bins) over primitive references.
//   * Big tasks (nodes of more than kSmallMax references) go level by level,
//     three launches a level. k_bin: blocks of kChunk references with
//     shared-memory bins, merged into per-task global bins. k_split: one block
//     per task picks the split plane, places the task's chunks and creates the
//     children. k_scatter: the stable partition by chunk, which also gathers
//     the children's centroid bounds.
//   * A node of at most kSmallMax references is finished by one block in
//     shared memory (k_subtree): every level below it, the leaves, and the
//     collapse's cost program over the subtree.
// Node ids and the order of the task lists depend on scheduling; the tree, the
// order of the references in its leaves and everything derived from them do
// not (float min/max merges, integer counts and stable partitions are order
// independent), so a build is a pure function of its input.
//
// Wide phase: breadth-first collapse to 8 slots, two launches a level, eight
// lanes per wide node, 16-bit child boxes, octant-ordered slots, triangle
// records in leaf order (src/accelerators/wide_bvh.cpp:430-472 packs TriangleN
// likewise). Which binary nodes fill a wide node's slots is chosen either
//   * SAH-optimally (the default): a bottom-up dynamic program over the
//     binary tree gives every node its least SAH cost when it may occupy
//     1..8 slots of its parent (the method of Ylitie, Karras and Laine,
//     "Efficient Incoherent Ray Traversal on GPUs Through Compressed Wide
//     BVHs", HPG 2017, restated for leaves of at most 3 triangles), and the
//     collapse follows its choices; or
//   * greedily, as the reference does (src/accelerators/wide_bvh.cpp:200-243):
//     open the internal child of largest surface area until 8 slots are used.
//
// Every count stays in device memory, so a build is a fixed sequence of
// launches that waits on nothing. build() enqueues the levels it expects and
// reads the counters back once, at the end (it continues where they fell
// short); enqueue() captures the sequence in a CUDA graph.
#include "build.cuh"

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdio>
#include <cstring>

namespace ag {
namespace {

constexpr uint32_t kSmallMax = 512;  // nodes up to this size are finished by one block
constexpr uint32_t kChunk = 1024;    // references per block of a big task
constexpr int kChunkThreads = 256;   // kChunk / 4
constexpr int kBinWords = 7;         // lo3 hi3 count
constexpr int kAxisBinWords = kSahBins * kBinWords;
constexpr int kTaskBinWords = 3 * kAxisBinWords;
constexpr int kChunkCounts = 3 * kSahBins;
constexpr uint32_t kMaxLevels = 1024;
constexpr uint32_t kMaxWideLevels = 64;

// A big task. The centroid bounds are order-preserving integers (f2ord),
// gathered by the parent's k_scatter.
struct alignas(16) BigTask {
    uint32_t clo[3];
    uint32_t node;
    uint32_t chi[3];
    uint32_t begin;
    uint32_t count;
    uint32_t chunk0;  // its first entry of the level's chunk list
    uint32_t pad[2];
};

struct BigSplit {
    int axis;
    int bin;
    int mode;  // 0 = SAH bin split, 1 = median (all centroids coincide, or every cost overflows)
    uint32_t nL;
    uint32_t child[2];  // big-task index of each child in the next level, kNoTask for a small one
};
constexpr uint32_t kNoTask = 0xffffffffu;

// A node of at most kSmallMax references, finished by k_subtree.
struct SmallTask {
    uint32_t node, begin, count, level;
};

// Counter words. The kLevel* arrays hold one word per binary level, the
// kWide* arrays one per collapse level.
enum Counter {
    kCntBounds = 0,        // 12 words: box and centroid bounds of all primitives (f2ord)
    kCntNodes = 12,        // binary node ids handed out
    kCntRealNodes,         // binary nodes of the tree (id ranges of subtrees have gaps)
    kCntSmall,             // entries of the small-task list
    kCntTicket,            // next small task to be taken by k_subtree
    kCntLevels,            // binary levels
    kCntFailed,            // kFail* bits: the tree was not finished; the collapse is skipped
    kCntSlots,             // filled child slots
    kCntRootAreaInv,       // float bits: 1 / half-area of the root box
    kCntSah,               // float bits: SAH cost of the wide tree
    kCntWords = 32
};
constexpr uint32_t kLevelBig = kCntWords;                             // big tasks
constexpr uint32_t kLevelChunks = kLevelBig + kMaxLevels + 2;         // their chunks
constexpr uint32_t kLevelNodes = kLevelChunks + kMaxLevels + 2;       // first node id
constexpr uint32_t kWideItems = kLevelNodes + kMaxLevels + 2;         // wide nodes of the level
constexpr uint32_t kWideTris = kWideItems + kMaxWideLevels + 2;       // triangle records placed by the level
constexpr uint32_t kWideNodeBase = kWideTris + kMaxWideLevels + 2;    // first wide node of the next level
constexpr uint32_t kWideTriBase = kWideNodeBase + kMaxWideLevels + 2; // first triangle record of the level
constexpr uint32_t kFailLevels = 1u;    // big tasks left after the levels run, or a tree deeper than the cap
constexpr uint32_t kFailCapacity = 2u;  // a list was full (never in a consistent build)
constexpr uint32_t kAllWords = kWideTriBase + kMaxWideLevels + 2;

// --------------------------------------------------------------------------
// Binning arithmetic. Every kernel must compute identical bin indices, so all
// float operations are explicitly rounded (no contraction into FMA).
AG_D float centroid(float lo, float hi) { return __fmul_rn(0.5f, __fadd_rn(lo, hi)); }
AG_D float axis_scale(float clo, float chi)
{
    float e = __fsub_rn(chi, clo);
    return e > 0.0f ? __fdiv_rn(float(kSahBins), e) : 0.0f;
}
AG_D int bin_of(float c, float clo, float scale)
{
    int b = __float2int_rz(__fmul_rn(__fsub_rn(c, clo), scale));
    return min(max(b, 0), kSahBins - 1);
}

AG_D void bin_init_word(uint32_t* w, int k)
{
    *w = k % kBinWords < 3 ? 0xffffffffu : 0u;  // min words start at the largest key, max words and counts at 0
}

// Half area of a box and the SAH cost of a split. Explicitly rounded, so that
// every kernel that evaluates the same split gets the same cost.
AG_D float area_of(float lx, float ly, float lz, float hx, float hy, float hz)
{
    const float ex = __fsub_rn(hx, lx), ey = __fsub_rn(hy, ly), ez = __fsub_rn(hz, lz);
    return __fmaf_rn(ez, ex, __fmaf_rn(ey, ez, __fmul_rn(ex, ey)));
}
AG_D float split_cost(uint32_t nL, float areaL, uint32_t nR, float areaR)
{
    return __fmaf_rn(float(nR), areaR, __fmul_rn(float(nL), areaL));
}

// Inclusive warp scans for union-of-boxes and counts.
template <bool kForward>
AG_D float scan_min(float v)
{
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        float y = kForward ? __shfl_up_sync(0xffffffffu, v, o) : __shfl_down_sync(0xffffffffu, v, o);
        bool ok = kForward ? (lane_id() >= (uint32_t)o) : (lane_id() + o < 32);
        if (ok) v = fminf(v, y);
    }
    return v;
}
template <bool kForward>
AG_D float scan_max(float v)
{
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        float y = kForward ? __shfl_up_sync(0xffffffffu, v, o) : __shfl_down_sync(0xffffffffu, v, o);
        bool ok = kForward ? (lane_id() >= (uint32_t)o) : (lane_id() + o < 32);
        if (ok) v = fmaxf(v, y);
    }
    return v;
}
AG_D uint32_t scan_add(uint32_t v)
{
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, v, o);
        if (lane_id() >= (uint32_t)o) v += y;
    }
    return v;
}

// Result of a warp-wide split search over the bins of one task.
struct SplitChoice {
    float cost;
    int axis;
    int bin;
    uint32_t nL;
    float L[6];  // lo3 hi3 of the left child
    float R[6];
};

AG_D void split_reset(SplitChoice& c)
{
    c.cost = FLT_MAX;
    c.axis = -1;
    c.bin = 0;
    c.nL = 0;
}

// Evaluate all 31 split planes of one axis from bins held one per lane
// (lane = bin). `v` holds the lane's bin: lo3 hi3 as floats (empty bins:
// lo = +FLT_MAX, hi = -FLT_MAX) and `cnt`; total is the task's count. Updates
// `best` when a cheaper split is found (ties keep the earlier axis / lower bin).
AG_D void eval_axis(int axis, const float v[6], uint32_t cnt, uint32_t total, SplitChoice& best)
{
    float Lv[6], Rn[6];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        Lv[k] = scan_min<true>(v[k]);
        Lv[3 + k] = scan_max<true>(v[3 + k]);
        // right side of the plane after bin k is bins k+1..31
        Rn[k] = __shfl_down_sync(0xffffffffu, scan_min<false>(v[k]), 1);
        Rn[3 + k] = __shfl_down_sync(0xffffffffu, scan_max<false>(v[3 + k]), 1);
    }
    const uint32_t cL = scan_add(cnt);
    const uint32_t cR = total - cL;
    float cost = FLT_MAX;
    if (lane_id() < 31 && cL > 0 && cR > 0)
        cost = split_cost(cL, area_of(Lv[0], Lv[1], Lv[2], Lv[3], Lv[4], Lv[5]), cR,
                          area_of(Rn[0], Rn[1], Rn[2], Rn[3], Rn[4], Rn[5]));
    // warp argmin (cost, then lowest lane)
    float bc = cost;
    int bl = (int)lane_id();
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        float oc = __shfl_xor_sync(0xffffffffu, bc, o);
        int ol = __shfl_xor_sync(0xffffffffu, bl, o);
        if (oc < bc || (oc == bc && ol < bl)) { bc = oc; bl = ol; }
    }
    if (bc < best.cost) {
        best.cost = bc;
        best.axis = axis;
        best.bin = bl;
        best.nL = __shfl_sync(0xffffffffu, cL, bl);
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            best.L[k] = __shfl_sync(0xffffffffu, Lv[k], bl);
            best.R[k] = __shfl_sync(0xffffffffu, Rn[k], bl);
        }
    }
}

AG_D void load_bin(const uint32_t* b, float v[6], uint32_t& cnt)
{
    cnt = b[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) v[k] = cnt ? ord2f(b[k]) : (k < 3 ? FLT_MAX : -FLT_MAX);
}

AG_D void bin_accumulate(uint32_t* bin, const uint32_t ord[6])
{
    atomicMin(bin + 0, ord[0]);
    atomicMin(bin + 1, ord[1]);
    atomicMin(bin + 2, ord[2]);
    atomicMax(bin + 3, ord[3]);
    atomicMax(bin + 4, ord[4]);
    atomicMax(bin + 5, ord[5]);
    atomicAdd(bin + 6, 1u);
}

// The same, for bins that many references fall into: a bound that the bin
// already covers needs no atomic. The bounds only ever widen, so a stale word
// costs an atomic and changes nothing.
AG_D void bin_widen(uint32_t* bin, const uint32_t ord[6])
{
    const volatile uint32_t* seen = bin;
    uint32_t w[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) w[k] = seen[k];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        if (ord[k] < w[k]) atomicMin(bin + k, ord[k]);
        if (ord[3 + k] > w[3 + k]) atomicMax(bin + 3 + k, ord[3 + k]);
    }
    atomicAdd(bin + 6, 1u);
}

// Primitive boxes: {lo.xyz, hi.x}, {hi.y, hi.z, 0, 0}, one 32-byte sector each.
AG_D void load_box(const float4* boxes, uint32_t p, float lo[3], float hi[3])
{
    const float4 a = boxes[2ull * p];
    const float2 b = *reinterpret_cast<const float2*>(boxes + 2ull * p + 1);
    lo[0] = a.x; lo[1] = a.y; lo[2] = a.z;
    hi[0] = a.w; hi[1] = b.x; hi[2] = b.y;
}

AG_D void write_node(BinNode* bnodes, uint32_t id, const float box[6], uint32_t begin, uint32_t count)
{
    BinNode b;
    b.lo = mk3(box[0], box[1], box[2]);
    b.hi = mk3(box[3], box[4], box[5]);
    b.begin = begin;
    b.count = count;
    b.left = -1;
    b.right = -1;
    b.pad[0] = b.pad[1] = 0u;
    bnodes[id] = b;
}

// --------------------------------------------------------------------------
// The kernels of a build form a chain in which each needs all of the one
// before it, 30 to 70 launches of which many run for a few microseconds. They
// are launched with programmatic stream serialisation: the blocks of the next
// kernel are placed while this one runs, and chain_wait(), the first statement
// of every kernel of the chain in every thread, holds them until it has
// finished and its writes are visible. Only then is the kernel after them
// allowed in, so at most one is waiting at a time, and each kernel's end
// implies the end of all before it. The pointers of these kernels carry no
// __restrict__: it would let the compiler take what the kernel before writes
// for constant data. 1M triangles: 2,091 to 1,995 us; an animated frame of 8k
// triangles: 488 to 404 us (B200).
AG_D void chain_allow() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
AG_D void chain_wait()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    chain_allow();
}

// --------------------------------------------------------------------------
// Preparation: counters, primitive boxes and root bounds.
__global__ void k_begin(uint32_t* cnt)
{
    chain_allow();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < kAllWords; i += gridDim.x * blockDim.x)
        cnt[i] = (i < 3 || (i >= 6 && i < 9)) ? 0xffffffffu : 0u;  // the bounds' min words, else 0
}

// Primitives 0 .. ntris-1 are triangles, ntris .. n-1 spheres (centre +
// radius): their box is centre -+ radius. The root's bounds are reduced per
// block before the 12 atomics: one set of atomics per warp took 256 of the
// 262 us of this kernel on 1M triangles.
constexpr int kPrepThreads = 256;
__global__ void __launch_bounds__(kPrepThreads) k_prep_prims(const float* verts,
                                                             const uint32_t* idx, uint32_t ntris,
                                                             const float4* spheres, uint32_t n,
                                                             float4* boxes, uint32_t* refs,
                                                             uint32_t* bounds)
{
    chain_wait();
    __shared__ uint32_t sb[12];
    if (threadIdx.x < 12) sb[threadIdx.x] = (threadIdx.x < 3 || (threadIdx.x >= 6 && threadIdx.x < 9)) ? 0xffffffffu : 0u;
    __syncthreads();
    float lo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, hi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
    float c[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, cmx[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
    for (uint32_t i = blockIdx.x * kPrepThreads + threadIdx.x; i < n; i += gridDim.x * kPrepThreads) {
        float l[3], h[3];
        if (i < ntris) {
            const uint32_t* t = idx + 3ull * i;
            float p[3][3];
#pragma unroll
            for (int v = 0; v < 3; ++v)
#pragma unroll
                for (int k = 0; k < 3; ++k) p[v][k] = verts[3ull * t[v] + k];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                l[k] = fminf(fminf(p[0][k], p[1][k]), p[2][k]);
                h[k] = fmaxf(fmaxf(p[0][k], p[1][k]), p[2][k]);
            }
        } else {
            const float4 sp = spheres[i - ntris];
            const float r = fabsf(sp.w);
            l[0] = __fsub_rd(sp.x, r); l[1] = __fsub_rd(sp.y, r); l[2] = __fsub_rd(sp.z, r);
            h[0] = __fadd_ru(sp.x, r); h[1] = __fadd_ru(sp.y, r); h[2] = __fadd_ru(sp.z, r);
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float ck = centroid(l[k], h[k]);
            lo[k] = fminf(lo[k], l[k]);
            hi[k] = fmaxf(hi[k], h[k]);
            c[k] = fminf(c[k], ck);
            cmx[k] = fmaxf(cmx[k], ck);
        }
        boxes[2ull * i] = make_float4(l[0], l[1], l[2], h[0]);
        boxes[2ull * i + 1] = make_float4(h[1], h[2], 0.0f, 0.0f);
        refs[i] = i;
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const uint32_t a = __reduce_min_sync(0xffffffffu, f2ord(lo[k])), b = __reduce_max_sync(0xffffffffu, f2ord(hi[k]));
        const uint32_t d = __reduce_min_sync(0xffffffffu, f2ord(c[k])), e = __reduce_max_sync(0xffffffffu, f2ord(cmx[k]));
        if (lane_id() == 0) {
            atomicMin(sb + k, a);
            atomicMax(sb + 3 + k, b);
            atomicMin(sb + 6 + k, d);
            atomicMax(sb + 9 + k, e);
        }
    }
    __syncthreads();
    const uint32_t w = threadIdx.x;
    if (w < 12) {
        if (w < 3 || (w >= 6 && w < 9)) atomicMin(bounds + w, sb[w]);
        else atomicMax(bounds + w, sb[w]);
    }
}

__global__ void k_root(uint32_t n, uint32_t* cnt, BigTask* big, BinNode* bnodes,
                       SmallTask* small, uint32_t* chunkTask, uint32_t* bins)
{
    chain_wait();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t chunks = n > kSmallMax ? (n + kChunk - 1) / kChunk : 0u;
    if (i == 0) {
        const uint32_t* bounds = cnt + kCntBounds;
        float box[6];
        for (int k = 0; k < 6; ++k) box[k] = ord2f(bounds[k]);
        write_node(bnodes, 0, box, 0, n);
        if (chunks) {
            BigTask t{};
            for (int k = 0; k < 3; ++k) {
                t.clo[k] = bounds[6 + k];
                t.chi[k] = bounds[9 + k];
            }
            t.node = 0;
            t.begin = 0;
            t.count = n;
            t.chunk0 = 0;
            big[0] = t;
        } else {
            small[0] = SmallTask{0u, 0u, n, 0u};
        }
        cnt[kLevelBig] = chunks ? 1u : 0u;
        cnt[kLevelChunks] = chunks;
        cnt[kCntSmall] = chunks ? 0u : 1u;
        cnt[kCntNodes] = 1u;
        cnt[kCntRealNodes] = 1u;
    }
    if (i < chunks) chunkTask[i] = 0;
    if (chunks && i < (uint32_t)kTaskBinWords) bin_init_word(bins + i, (int)i);
}

// --------------------------------------------------------------------------
// Big tasks, level by level. The lists are double-buffered by level parity.
// One block per chunk of 1,024 references; the chunk's bin counts are kept
// (16 bits each), so that k_split can place the chunks of the partition
// without another pass over the references. 21 atomics a reference on the
// shared bins bound it at first, and at the top the 1,024 blocks' merges into
// one task's bins: most of a bin's later references widen nothing, so a plain
// read comes before each atomic min / max, here and in the merge, and the four
// references of a thread are fetched together. Root of 1M triangles: 43 to
// 31 us, the level below 37 to 25 (B200).
__global__ void __launch_bounds__(kChunkThreads) k_bin(const BigTask* tasks, const uint32_t* refs,
                                                       const float4* boxes,
                                                       const uint32_t* chunkTask,
                                                       uint32_t* bins, uint16_t* chunkCnt,
                                                       uint32_t* cnt, uint32_t level, uint32_t capChunks)
{
    chain_wait();
    __shared__ uint32_t sb[kTaskBinWords];
    // the next level's nodes start where the ids handed out so far end
    if (blockIdx.x == 0 && threadIdx.x == 0) cnt[kLevelNodes + level + 1] = cnt[kCntNodes];
    const uint32_t nc = cnt[kCntFailed] ? 0u : min(cnt[kLevelChunks + level], capChunks);
    for (uint32_t cb = blockIdx.x; cb < nc; cb += gridDim.x) {
        for (int k = threadIdx.x; k < kTaskBinWords; k += kChunkThreads) bin_init_word(sb + k, k);
        __syncthreads();
        const uint32_t bi = chunkTask[cb];
        const BigTask task = tasks[bi];
        float clo[3], sc[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            clo[a] = ord2f(task.clo[a]);
            sc[a] = axis_scale(clo[a], ord2f(task.chi[a]));
        }
        const uint32_t begin = task.begin + (cb - task.chunk0) * kChunk, end = min(task.begin + task.count, begin + kChunk);
        uint32_t p[kChunk / kChunkThreads];
#pragma unroll
        for (int r = 0; r < (int)kChunk / kChunkThreads; ++r) {
            const uint32_t i = begin + r * kChunkThreads + threadIdx.x;
            p[r] = i < end ? refs[i] : kNoTask;
        }
#pragma unroll
        for (int r = 0; r < (int)kChunk / kChunkThreads; ++r) {
            if (p[r] == kNoTask) break;
            float lo[3], hi[3];
            load_box(boxes, p[r], lo, hi);
            uint32_t ord[6];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                ord[k] = f2ord(lo[k]);
                ord[3 + k] = f2ord(hi[k]);
            }
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                if (sc[a] == 0.0f) continue;
                bin_widen(sb + a * kAxisBinWords + bin_of(centroid(lo[a], hi[a]), clo[a], sc[a]) * kBinWords, ord);
            }
        }
        __syncthreads();
        uint32_t* g = bins + size_t(bi) * kTaskBinWords;
        for (int k = threadIdx.x; k < kTaskBinWords; k += kChunkThreads) {
            const int f = k % kBinWords;
            const uint32_t filled = sb[k - f + 6];
            if (f == 6) chunkCnt[size_t(cb) * kChunkCounts + k / kBinWords] = (uint16_t)filled;
            if (filled == 0) continue;  // empty bin: nothing to merge
            const uint32_t mine = sb[k], seen = __ldcg(g + k);
            if (f == 6) atomicAdd(g + k, filled);
            else if (f < 3 && mine < seen) atomicMin(g + k, mine);
            else if (f >= 3 && mine > seen) atomicMax(g + k, mine);
        }
        __syncthreads();  // sb is cleared again for the next chunk
    }
}

// One block per big task: the split (a warp per axis), the children, and the
// position of every chunk's left references in the partition.
constexpr int kSplitThreads = 256;
__global__ void __launch_bounds__(kSplitThreads) k_split(const BigTask* tasks, const uint32_t* bins,
                                                         const uint16_t* chunkCnt,
                                                         uint32_t* chunkLeft, BigSplit* splits,
                                                         BinNode* bnodes, BigTask* next,
                                                         uint32_t* nextChunkTask,
                                                         uint32_t* nextBins, SmallTask* small,
                                                         uint32_t* cnt, uint32_t level, uint32_t capBig,
                                                         uint32_t capChunks, uint32_t capPrims,
                                                         uint32_t* status)
{
    chain_wait();
    __shared__ SplitChoice axisBest[3];
    __shared__ BigSplit split;
    __shared__ uint32_t childChunk0[2], childChunks[2], warpSums[kSplitThreads / 32], failed;
    // (read by one thread: another block may set the flag, and the threads of a block stay together)
    if (threadIdx.x == 0) failed = cnt[kCntFailed] & kFailCapacity;
    __syncthreads();
    const uint32_t nb = failed ? 0u : min(cnt[kLevelBig + level], capBig);
    const uint32_t warp = threadIdx.x >> 5;
    for (uint32_t bi = blockIdx.x; bi < nb; bi += gridDim.x) {
        const BigTask task = tasks[bi];
        if (warp < 3) {
            SplitChoice best;
            split_reset(best);
            if (axis_scale(ord2f(task.clo[warp]), ord2f(task.chi[warp])) != 0.0f) {
                float v[6];
                uint32_t c;
                load_bin(bins + size_t(bi) * kTaskBinWords + warp * kAxisBinWords + lane_id() * kBinWords, v, c);
                eval_axis((int)warp, v, c, task.count, best);
            }
            if (lane_id() == 0) axisBest[warp] = best;
        }
        __syncthreads();
        if (threadIdx.x < 2) {  // lane k takes child k; the counters' round trips overlap
            const uint32_t k = threadIdx.x;
            SplitChoice best = axisBest[0];
#pragma unroll
            for (int a = 1; a < 3; ++a)
                if (axisBest[a].cost < best.cost) best = axisBest[a];
            const bool median = best.axis < 0;
            const uint32_t nL = median ? task.count / 2 : best.nL;
            const uint32_t begin = k ? task.begin + nL : task.begin, count = k ? task.count - nL : nL;
            const uint32_t chunks = count > kSmallMax ? (count + kChunk - 1) / kChunk : 0u;
            uint32_t id = 0, ci = kNoTask, c0 = 0, si = 0;
            if (k == 0) id = atomicAdd(cnt + kCntNodes, 2u);
            if (chunks) {
                ci = atomicAdd(cnt + kLevelBig + level + 1, 1u);
                c0 = atomicAdd(cnt + kLevelChunks + level + 1, chunks);
            } else {
                si = atomicAdd(cnt + kCntSmall, 1u);
            }
            if (k == 0) {
                atomicAdd(cnt + kCntRealNodes, 2u);
                atomicMax(cnt + kCntLevels, level + 1u);
            }
            float box[6];
#pragma unroll
            for (int j = 0; j < 6; ++j) box[j] = k ? best.R[j] : best.L[j];
            if (median) {  // no plane with a finite cost (all centroids coincide): split by position, the children keep the parent's box
                const BinNode parent = bnodes[task.node];
                box[0] = parent.lo.x; box[1] = parent.lo.y; box[2] = parent.lo.z;
                box[3] = parent.hi.x; box[4] = parent.hi.y; box[5] = parent.hi.z;
            }
            id = __shfl_sync(3u, id, 0);
            // capacities: never exceeded by a consistent build; checked so that
            // inconsistent input cannot write past the buffers
            const bool nodes = id + 1u < 2u * capPrims;
            const bool listed = chunks ? ci < capBig && c0 + chunks <= capChunks : si < capPrims;
            if (nodes) {
                if (k == 0) {
                    bnodes[task.node].left = (int32_t)id;
                    bnodes[task.node].right = (int32_t)id + 1;
                }
                write_node(bnodes, id + k, box, begin, count);
            }
            if (nodes && listed) {
                if (chunks) {
                    BigTask t{};
                    // gathered by k_scatter; a split by position of finite
                    // centroids starts from the parent's bounds, so that where
                    // the costs overflow (boxes beyond about 1e18) the halves
                    // are halved again, and the depth stays a balanced tree's
                    bool inherit = median;
                    for (int a = 0; a < 3; ++a)
                        inherit = inherit && isfinite(ord2f(task.clo[a])) && isfinite(ord2f(task.chi[a]));
                    for (int a = 0; a < 3; ++a) {
                        t.clo[a] = inherit ? task.clo[a] : 0xffffffffu;
                        t.chi[a] = inherit ? task.chi[a] : 0u;
                    }
                    t.node = id + k;
                    t.begin = begin;
                    t.count = count;
                    t.chunk0 = c0;
                    next[ci] = t;
                } else {
                    small[si] = SmallTask{id + k, begin, count, level + 1u};
                }
            } else {
                atomicOr(status, kErrBadIndex);
                atomicOr(cnt + kCntFailed, kFailCapacity);
            }
            const bool pass = nodes && listed && chunks;  // to the next level
            split.child[k] = pass ? ci : kNoTask;
            childChunk0[k] = c0;
            childChunks[k] = pass ? chunks : 0u;
            if (k == 0) {
                split.axis = median ? 0 : best.axis;
                split.bin = best.bin;
                split.mode = median ? 1 : 0;
                split.nL = nL;
            }
            __syncwarp(3u);
            if (k == 0) splits[bi] = split;
        }
        __syncthreads();
        const BigSplit s = split;
#pragma unroll
        for (int k = 0; k < 2; ++k)
            if (s.child[k] != kNoTask) {
                for (uint32_t c = threadIdx.x; c < childChunks[k]; c += kSplitThreads)
                    nextChunkTask[childChunk0[k] + c] = s.child[k];
                uint32_t* b = nextBins + size_t(s.child[k]) * kTaskBinWords;
                for (int w = threadIdx.x; w < kTaskBinWords; w += kSplitThreads) bin_init_word(b + w, w);
            }
        // left references before each chunk
        const uint32_t chunks = (task.count + kChunk - 1) / kChunk;
        uint32_t run = 0;
        for (uint32_t base = 0; base < chunks; base += kSplitThreads) {
            const uint32_t c = base + threadIdx.x;
            uint32_t left = 0;
            if (c < chunks && s.mode == 0) {
                // the row of the axis: 32 counts of 16 bits, 64 bytes
                const uint4* p = reinterpret_cast<const uint4*>(chunkCnt + size_t(task.chunk0 + c) * kChunkCounts + s.axis * kSahBins);
                uint4 q[kSahBins / 8];
#pragma unroll
                for (int k = 0; k < kSahBins / 8; ++k) q[k] = p[k];
#pragma unroll
                for (int k = 0; k < kSahBins / 8; ++k) {
                    const uint32_t v[4] = {q[k].x, q[k].y, q[k].z, q[k].w};
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int b = 8 * k + 2 * j;
                        left += (b <= s.bin ? v[j] & 0xffffu : 0u) + (b + 1 <= s.bin ? v[j] >> 16 : 0u);
                    }
                }
            }
            const uint32_t inc = scan_add(left);
            if (lane_id() == 31) warpSums[warp] = inc;
            __syncthreads();
            uint32_t before = 0, all = 0;
#pragma unroll
            for (uint32_t w = 0; w < kSplitThreads / 32; ++w) {
                if (w < warp) before += warpSums[w];
                all += warpSums[w];
            }
            if (c < chunks) chunkLeft[task.chunk0 + c] = s.mode == 0 ? run + before + inc - left : min(c * kChunk, s.nL);
            run += all;
            __syncthreads();  // warpSums is written again
        }
    }
}

// Stable partition, one block per chunk, four references a thread, a block's
// width apart: whole sectors of references, and a reference's rank is a ballot
// within its warp plus the counts of the 32 (round, warp) groups before it.
// Also the centroid bounds of the big children. Bound by the latency of
// reference -> box -> rank, so by the blocks in flight: 8 per SM hold the
// 1,024 chunks of 1M references at once. With four consecutive references a
// thread and 4 blocks per SM a level took 22 us, at 6 blocks 19 (B200).
constexpr int kScatterRounds = (int)kChunk / kChunkThreads;
static_assert(kScatterRounds * (kChunkThreads / 32) == 32, "one lane a group in the scan of the groups");
__global__ void __launch_bounds__(kChunkThreads, 8) k_scatter(BigTask* next, const BigTask* tasks,
                                                              const uint32_t* refs,
                                                              uint32_t* refsNext,
                                                              const float4* boxes,
                                                              const uint32_t* chunkTask,
                                                              const BigSplit* splits,
                                                              const uint32_t* chunkLeft,
                                                              const uint32_t* cnt, uint32_t level,
                                                              uint32_t capChunks, uint32_t* status)
{
    chain_wait();
    __shared__ uint32_t groupLeft[32], cb12[12];
    const uint32_t nc = cnt[kCntFailed] ? 0u : min(cnt[kLevelChunks + level], capChunks);
    const uint32_t warp = threadIdx.x >> 5;
    for (uint32_t cb = blockIdx.x; cb < nc; cb += gridDim.x) {
        const uint32_t bi = chunkTask[cb];
        const BigTask& task = tasks[bi];
        const BigSplit& s = splits[bi];
        const uint32_t taskBegin = task.begin, taskCount = task.count, nL = s.nL;
        const uint32_t first = (cb - task.chunk0) * kChunk;  // within the task
        const uint32_t count = min(taskCount - first, kChunk);
        const uint32_t leftBefore = chunkLeft[cb], rightBefore = first - leftBefore;
        const int axis = s.axis, bin = s.bin;
        const bool byPosition = s.mode == 1;
        const float clo = ord2f(task.clo[axis]);
        const float scale = axis_scale(clo, ord2f(task.chi[axis]));
        if (threadIdx.x < 12) cb12[threadIdx.x] = threadIdx.x % 6 < 3 ? 0xffffffffu : 0u;
        uint32_t p[kScatterRounds];
#pragma unroll
        for (int r = 0; r < kScatterRounds; ++r) {
            const uint32_t i = r * kChunkThreads + threadIdx.x;
            p[r] = i < count ? refs[taskBegin + first + i] : kNoTask;
        }
        uint32_t leftMask[kScatterRounds];
        uint32_t bb[12] = {0xffffffffu, 0xffffffffu, 0xffffffffu, 0u, 0u, 0u, 0xffffffffu, 0xffffffffu, 0xffffffffu, 0u, 0u, 0u};
#pragma unroll
        for (int r = 0; r < kScatterRounds; ++r) {
            bool left = false;
            if (p[r] != kNoTask) {
                float lo[3], hi[3];
                load_box(boxes, p[r], lo, hi);
                const float c[3] = {centroid(lo[0], hi[0]), centroid(lo[1], hi[1]), centroid(lo[2], hi[2])};
                const float ca = axis == 0 ? c[0] : (axis == 1 ? c[1] : c[2]);
                left = byPosition ? first + r * kChunkThreads + threadIdx.x < nL : bin_of(ca, clo, scale) <= bin;
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    const uint32_t o = f2ord(c[a]);
                    if (left) {
                        bb[a] = min(bb[a], o);
                        bb[3 + a] = max(bb[3 + a], o);
                    } else {
                        bb[6 + a] = min(bb[6 + a], o);
                        bb[9 + a] = max(bb[9 + a], o);
                    }
                }
            }
            leftMask[r] = __ballot_sync(0xffffffffu, left);
            if (lane_id() == 0) groupLeft[r * (kChunkThreads / 32) + warp] = __popc(leftMask[r]);
        }
        __syncthreads();
        const uint32_t mine = groupLeft[lane_id()], before = scan_add(mine) - mine;
#pragma unroll
        for (int r = 0; r < kScatterRounds; ++r) {
            const uint32_t leftRank = __shfl_sync(0xffffffffu, before, r * (kChunkThreads / 32) + (int)warp) +
                                      __popc(leftMask[r] & ((1u << lane_id()) - 1u));
            if (p[r] == kNoTask) continue;
            const uint32_t i = r * kChunkThreads + threadIdx.x;
            const uint32_t at = leftMask[r] >> lane_id() & 1u ? leftBefore + leftRank : nL + rightBefore + i - leftRank;
            if (at >= taskCount) { atomicOr(status, kErrBadIndex); continue; }
            refsNext[taskBegin + at] = p[r];
        }
        const uint32_t child[2] = {s.child[0], s.child[1]};
#pragma unroll
        for (int side = 0; side < 2; ++side) {
            if (child[side] == kNoTask) continue;
#pragma unroll
            for (int a = 0; a < 6; ++a) {
                const uint32_t v = a < 3 ? __reduce_min_sync(0xffffffffu, bb[6 * side + a])
                                         : __reduce_max_sync(0xffffffffu, bb[6 * side + a]);
                if (lane_id() == 0) {
                    if (a < 3) atomicMin(cb12 + 6 * side + a, v);
                    else atomicMax(cb12 + 6 * side + a, v);
                }
            }
        }
        __syncthreads();
        const uint32_t w = threadIdx.x, to = w < 6 ? child[0] : child[1];
        if (w < 12 && to != kNoTask) {
            BigTask* t = next + to;
            if (w % 6 < 3) atomicMin(t->clo + w % 6, cb12[w]);
            else atomicMax(t->chi + w % 6 - 3, cb12[w]);
        }
        __syncthreads();  // the shared words are written again for the next chunk
    }
}

// --------------------------------------------------------------------------
// SAH cost program of the collapse. For binary node x of area A, count n and
// children l, r:
//   leaf(x)    = A * triCost * n                       (n <= kMaxLeafTris)
//   D(x, j)    = min over k in 1..j-1 of C(l, k) + C(r, j - k)
//   C(x, 1)    = leaf(x) if n <= kMaxLeafTris, else A + D(x, 8)  (x in one slot:
//                a leaf, or an internal child whose own wide node tests 8 slots)
//   C(x, j)    = min(C(x, j - 1), D(x, j))             (x spread over at most j slots)
// with a wide-node visit costing 1 per unit area. C[j - 1] holds C(x, j) for
// j = 1..7; nibble j - 1 of the choice holds the k of D(x, j) when it was
// taken (0: x keeps j - 1 slots; nibble 7: the split of x's own wide node). A
// binary leaf costs leaf(x) for every j.
constexpr int kCosts = 7;
AG_D float leaf_cost(float area, uint32_t count, float triCost)
{
    return count <= (uint32_t)kMaxLeafTris ? __fmul_rn(__fmul_rn(area, triCost), float(count)) : INFINITY;
}
AG_D uint32_t collapse_cost(const float L[kCosts], const float R[kCosts], float A, uint32_t count, float triCost,
                            float C[kCosts])
{
    float D[9];
    uint32_t K[9];
#pragma unroll
    for (int j = 2; j <= 8; ++j) {
        float best = INFINITY;
        uint32_t bk = 1;
#pragma unroll
        for (int k = 1; k < j; ++k) {
            const float v = __fadd_rn(L[k - 1], R[j - k - 1]);
            if (v < best) {
                best = v;
                bk = (uint32_t)k;
            }
        }
        D[j] = best;
        K[j] = bk;
    }
    float prev = count <= (uint32_t)kMaxLeafTris ? leaf_cost(A, count, triCost) : __fadd_rn(A, D[8]);
    C[0] = prev;
    uint32_t ch = K[8] << 28;
#pragma unroll
    for (int j = 2; j <= 7; ++j) {
        if (D[j] < prev) {
            prev = D[j];
            ch |= K[j] << (4 * (j - 1));
        }
        C[j - 1] = prev;
    }
    return ch;
}

// --------------------------------------------------------------------------
// Small nodes: one block finishes the subtree of a node of at most kSmallMax
// references in shared memory: every split below it, the leaves, the order of
// its references, and its part of the cost program. Against one launch (and
// its counts, scans and compaction) per level this removed half of a build's
// time and most of its launches.
//
// One thread per reference; the references' boxes move with the partition, so
// that a node's are consecutive. Nodes above kDirectMax references are split
// with shared-memory bins, kBinNodes of them at a time, a warp per node and
// axis for the search. The others are split without bins: a thread takes the
// plane after its own reference's bin as its candidate on each axis, sums the
// two sides over the node's references, and the node's cheapest candidate
// wins (a 64-bit shared-memory minimum over cost, axis, bin). Planes between
// two references' bins need no candidate of their own: they cut the same sets
// as the plane after the lower bin, which the bin search prefers as well. At
// eight references this takes about 400 instructions for four nodes; the bin
// search takes 1,500 for each.
//
// The kernel is a chain of short steps between block barriers, about 12 levels
// deep, and its time on a small scene is that chain's.
constexpr int kSubThreads = (int)kSmallMax;
constexpr uint32_t kSubWarps = kSubThreads / 32;
constexpr uint32_t kDirectMax = 32;
constexpr uint32_t kBinNodes = 8;
constexpr uint32_t kNoChild = 0xffffu;

struct SubSmem {
    float4 pa[kSmallMax];               // per position: lo.xyz, hi.x
    float4 pb[kSmallMax];               // hi.y, hi.z, bits: bins on the three axes and which have an extent, primitive id
    unsigned long long key[kSmallMax];  // per node of the level: its cheapest candidate
    union {
        uint32_t bins[kBinNodes][kTaskBinWords];
        float cost[(kSmallMax - 1) * kCosts];  // per internal node, once the tree is built
    };
    SplitChoice axisBest[kBinNodes][3];
    uint32_t cbounds[kBinNodes][6];     // centroid bounds (f2ord) of the nodes being binned
    float area[2 * kSmallMax];          // per node of the subtree
    uint32_t leftBits[kSmallMax / 32];
    uint32_t ticket, idBase, nodeTop, levelEnd, binCount;
    uint16_t binNode[kSmallMax / kDirectMax];  // the level's nodes above kDirectMax references
    uint16_t binSlot[kSmallMax];        // per node of the level: its entry there
    uint16_t posNode[kSmallMax];        // per position: the node it belongs to
    uint16_t begin[2 * kSmallMax], count[2 * kSmallMax], left[2 * kSmallMax];
    uint16_t levelStart[kSmallMax + 2];
};

AG_D void sub_box(const float4& a, const float4& b, float lo[3], float hi[3])
{
    lo[0] = a.x; lo[1] = a.y; lo[2] = a.z;
    hi[0] = a.w; hi[1] = b.x; hi[2] = b.y;
}
AG_D void box_reset(float b[6])
{
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        b[k] = FLT_MAX;
        b[3 + k] = -FLT_MAX;
    }
}
AG_D void box_add(float b[6], const float lo[3], const float hi[3])
{
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        b[k] = fminf(b[k], lo[k]);
        b[3 + k] = fmaxf(b[3 + k], hi[k]);
    }
}

// A node's split as its key: cost, axis, bin, candidate's position.
AG_D unsigned long long split_key(float cost, uint32_t axis, uint32_t bin, uint32_t p)
{
    return ((unsigned long long)__float_as_uint(cost) << 32) | (axis << 24) | (bin << 16) | p;
}
constexpr unsigned long long kNoSplit = ~0ull;  // all centroids coincide: split by position
AG_D bool key_left(unsigned long long key, uint32_t pbin, uint32_t local, uint32_t count)
{
    if (key == kNoSplit) return local < count / 2u;
    return ((pbin >> (8u * ((uint32_t)(key >> 24) & 0xffu))) & 0xffu) <= ((uint32_t)(key >> 16) & 0xffu);
}

// Two children of node nd (nL of its references go left). The subtree's nodes
// are 0 (the root, id rootNode) and 1, 2, ... (ids idBase, idBase + 1, ...).
AG_D void sub_children(SubSmem& s, BinNode* bnodes, uint32_t rootNode, uint32_t globalBegin, uint32_t nd,
                       uint32_t nL, const float L[6], const float R[6])
{
    const uint32_t ch = atomicAdd(&s.nodeTop, 2u);
    const uint32_t b = s.begin[nd], n = s.count[nd];
    s.left[nd] = (uint16_t)ch;
    s.begin[ch] = (uint16_t)b;
    s.count[ch] = (uint16_t)nL;
    s.left[ch] = (uint16_t)kNoChild;
    s.area[ch] = area_of(L[0], L[1], L[2], L[3], L[4], L[5]);
    s.begin[ch + 1] = (uint16_t)(b + nL);
    s.count[ch + 1] = (uint16_t)(n - nL);
    s.left[ch + 1] = (uint16_t)kNoChild;
    s.area[ch + 1] = area_of(R[0], R[1], R[2], R[3], R[4], R[5]);
    const uint32_t id = s.idBase + ch - 1, parent = nd == 0 ? rootNode : s.idBase + nd - 1;
    bnodes[parent].left = (int32_t)id;
    bnodes[parent].right = (int32_t)id + 1;
    write_node(bnodes, id, L, globalBegin + b, nL);
    write_node(bnodes, id + 1, R, globalBegin + b + nL, n - nL);
}

// Boxes of the two halves of a node whose centroids coincide.
AG_D void median_boxes(const SubSmem& s, uint32_t b, uint32_t c, float L[6], float R[6])
{
    box_reset(L);
    box_reset(R);
    for (uint32_t i = 0; i < c; ++i) {
        float lo[3], hi[3];
        sub_box(s.pa[b + i], s.pb[b + i], lo, hi);
        if (i < c / 2u) box_add(L, lo, hi);
        else box_add(R, lo, hi);
    }
}

// Splits the level's nodes above kDirectMax references (binNode). bin: this
// thread's entry of the list, kNoTask if it has none. Called by the whole block.
AG_D void sub_split_bins(SubSmem& s, BinNode* bnodes, uint32_t rootNode, uint32_t globalBegin, uint32_t ls,
                         uint32_t bin)
{
    const uint32_t tid = threadIdx.x, warp = tid >> 5, total = s.binCount;
    for (uint32_t first = 0; first < total; first += kBinNodes) {
        const uint32_t nodes = min(kBinNodes, total - first);
        const bool mine = bin - first < nodes;  // (wraps for kNoTask and entries of other rounds)
        const uint32_t slot = mine ? bin - first : 0u;
        for (uint32_t k = tid; k < nodes * kTaskBinWords; k += kSubThreads) bin_init_word(&s.bins[0][0] + k, (int)k);
        if (tid < nodes * 6) (&s.cbounds[0][0])[tid] = tid % 6 < 3 ? 0xffffffffu : 0u;
        __syncthreads();
        float lo[3], hi[3], c[3] = {0.0f, 0.0f, 0.0f};
        uint32_t cmin[3], cmax[3];
        sub_box(s.pa[tid], s.pb[tid], lo, hi);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            c[k] = centroid(lo[k], hi[k]);
            const bool nan = c[k] != c[k];  // no bound, as with fminf / fmaxf
            cmin[k] = nan ? f2ord(FLT_MAX) : f2ord(c[k]);
            cmax[k] = nan ? f2ord(-FLT_MAX) : f2ord(c[k]);
        }
        const uint32_t slot0 = __shfl_sync(0xffffffffu, slot, 0);
        if (__all_sync(0xffffffffu, mine && slot == slot0)) {  // one set of atomics for the warp
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const uint32_t a = __reduce_min_sync(0xffffffffu, cmin[k]), b = __reduce_max_sync(0xffffffffu, cmax[k]);
                if (lane_id() == 0) {
                    atomicMin(&s.cbounds[slot][k], a);
                    atomicMax(&s.cbounds[slot][3 + k], b);
                }
            }
        } else if (mine) {
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                atomicMin(&s.cbounds[slot][k], cmin[k]);
                atomicMax(&s.cbounds[slot][3 + k], cmax[k]);
            }
        }
        __syncthreads();
        if (mine) {
            uint32_t ord[6], v = 0;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                ord[k] = f2ord(lo[k]);
                ord[3 + k] = f2ord(hi[k]);
            }
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const float clo = ord2f(s.cbounds[slot][k]), sc = axis_scale(clo, ord2f(s.cbounds[slot][3 + k]));
                if (sc == 0.0f) continue;
                const uint32_t bk = (uint32_t)bin_of(c[k], clo, sc);
                v |= (bk << (8 * k)) | (1u << (24 + k));
                bin_accumulate(&s.bins[slot][k * kAxisBinWords + bk * kBinWords], ord);
            }
            s.pb[tid].z = __uint_as_float(v);
        }
        __syncthreads();
        for (uint32_t pair = warp; pair < nodes * 3u; pair += kSubWarps) {
            const uint32_t sl = pair / 3u, a = pair % 3u;
            SplitChoice best;
            split_reset(best);
            if (axis_scale(ord2f(s.cbounds[sl][a]), ord2f(s.cbounds[sl][3 + a])) != 0.0f) {
                float v[6];
                uint32_t n;
                load_bin(&s.bins[sl][a * kAxisBinWords + lane_id() * kBinWords], v, n);
                eval_axis((int)a, v, n, s.count[s.binNode[first + sl]], best);
            }
            if (lane_id() == 0) s.axisBest[sl][a] = best;
        }
        __syncthreads();
        if (lane_id() == 0 && warp < nodes) {  // a warp per node, so that their memory waits overlap
            const uint32_t nd = s.binNode[first + warp];
            int a = 0;
            for (int k = 1; k < 3; ++k)
                if (s.axisBest[warp][k].cost < s.axisBest[warp][a].cost) a = k;
            const SplitChoice& best = s.axisBest[warp][a];
            if (best.axis >= 0) {
                s.key[nd - ls] = split_key(best.cost, (uint32_t)best.axis, (uint32_t)best.bin, 0u);
                sub_children(s, bnodes, rootNode, globalBegin, nd, best.nL, best.L, best.R);
            } else {
                float L[6], R[6];
                median_boxes(s, s.begin[nd], s.count[nd], L, R);
                sub_children(s, bnodes, rootNode, globalBegin, nd, s.count[nd] / 2u, L, R);
            }
        }
        __syncthreads();  // the bins are cleared again for the next nodes
    }
}

// levels: the binary levels that the big-task kernels ran; big tasks left
// after them mean that the tree cannot be finished here (kCntFailed).
__global__ void __launch_bounds__(kSubThreads, 2) k_subtree(const SmallTask* small,
                                                            const uint32_t* refs0,
                                                            const uint32_t* refs1,
                                                            const float4* boxes,
                                                            BinNode* bnodes, uint32_t* order,
                                                            float* cost, uint32_t* choice,
                                                            float triCost, bool sah, uint32_t* cnt,
                                                            uint32_t levels, uint32_t capPrims)
{
    chain_wait();
    extern __shared__ __align__(16) unsigned char smem[];
    SubSmem& s = *reinterpret_cast<SubSmem*>(smem);
    const uint32_t tid = threadIdx.x;
    if (cnt[kLevelBig + levels] != 0u) {
        if (blockIdx.x == 0 && tid == 0) atomicOr(cnt + kCntFailed, kFailLevels);
        return;
    }
    const uint32_t numSmall = min(cnt[kCntSmall], capPrims);
    for (;;) {
        // (one thread reads the flag, which another block may set: the threads of a block stay together)
        if (tid == 0) s.ticket = cnt[kCntFailed] & kFailCapacity ? kNoTask : atomicAdd(cnt + kCntTicket, 1u);
        __syncthreads();
        const uint32_t ticket = s.ticket;
        if (ticket >= numSmall) break;
        const SmallTask task = small[ticket];
        const uint32_t n = min(task.count, kSmallMax), b0 = task.begin;
        const bool live = tid < n;  // this thread has a position
        if (live) {
            const uint32_t prim = ((task.level & 1u) ? refs1 : refs0)[b0 + tid];
            const float4 a = boxes[2ull * prim], b = boxes[2ull * prim + 1];
            s.pa[tid] = a;
            s.pb[tid] = make_float4(b.x, b.y, 0.0f, __uint_as_float(prim));
            s.posNode[tid] = 0;
        }
        if (tid == 0) {
            // ids of the 2 n - 2 nodes below the root (fewer are used when leaves hold several references)
            s.idBase = n > 1 ? atomicAdd(cnt + kCntNodes, 2u * n - 2u) : 0u;
            s.nodeTop = 1;
            s.begin[0] = 0;
            s.count[0] = (uint16_t)n;
            s.left[0] = (uint16_t)kNoChild;
            const BinNode r = bnodes[task.node];
            s.area[0] = area_of(r.lo.x, r.lo.y, r.lo.z, r.hi.x, r.hi.y, r.hi.z);
            s.binCount = 0;
        }
        __syncthreads();
        if (s.idBase + 2u * n - 2u > 2u * capPrims) {  // never in a consistent build
            if (tid == 0) atomicOr(cnt + kCntFailed, kFailCapacity);
            __syncthreads();
            continue;
        }
        uint32_t ls = 0, le = 1, lev = 0;
        while (ls < le) {
            if (tid == 0) s.levelStart[lev] = (uint16_t)ls;
            uint32_t nd = 0, c = 0, b = 0;
            if (live) {
                nd = s.posNode[tid];
                c = s.count[nd];
                b = s.begin[nd];
            }
            const bool active = live && nd >= ls && c >= 2u, direct = active && c <= kDirectMax;
            if (active && tid == b) {
                s.key[nd - ls] = kNoSplit;
                if (!direct) {
                    const uint32_t at = atomicAdd(&s.binCount, 1u);
                    s.binNode[at] = (uint16_t)nd;
                    s.binSlot[nd - ls] = (uint16_t)at;
                }
            }
            if (direct) {  // this reference's bins
                float clo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, chi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX}, lo[3], hi[3];
                for (uint32_t i = b; i < b + c; ++i) {
                    sub_box(s.pa[i], s.pb[i], lo, hi);
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        const float ck = centroid(lo[k], hi[k]);
                        clo[k] = fminf(clo[k], ck);
                        chi[k] = fmaxf(chi[k], ck);
                    }
                }
                sub_box(s.pa[tid], s.pb[tid], lo, hi);
                uint32_t v = 0;
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const float sc = axis_scale(clo[k], chi[k]);
                    if (sc != 0.0f) v |= ((uint32_t)bin_of(centroid(lo[k], hi[k]), clo[k], sc) << (8 * k)) | (1u << (24 + k));
                }
                s.pb[tid].z = __uint_as_float(v);
            }
            __syncthreads();
            if (s.binCount) sub_split_bins(s, bnodes, task.node, b0, ls, active && !direct ? s.binSlot[nd - ls] : kNoTask);
            // this reference's candidate planes; the best one's two sides stay in registers
            float bestL[6], bestR[6];
            uint32_t bestN = 0;
            unsigned long long key = kNoSplit;
            if (direct) {
                const uint32_t own = __float_as_uint(s.pb[tid].z);
                float bestCost = FLT_MAX;
#pragma unroll 1
                for (uint32_t a = 0; a < 3; ++a) {
                    if (!(own & (1u << (24 + a)))) continue;
                    const uint32_t sh = 8u * a, ob = (own >> sh) & 0xffu;
                    float L[6], R[6];
                    uint32_t nL = 0;
                    box_reset(L);
                    box_reset(R);
                    for (uint32_t i = b; i < b + c; ++i) {
                        const float4 pa = s.pa[i], pb = s.pb[i];
                        float lo[3], hi[3];
                        sub_box(pa, pb, lo, hi);
                        if (((__float_as_uint(pb.z) >> sh) & 0xffu) <= ob) {
                            box_add(L, lo, hi);
                            ++nL;
                        } else {
                            box_add(R, lo, hi);
                        }
                    }
                    if (nL >= c) continue;
                    const float sc = split_cost(nL, area_of(L[0], L[1], L[2], L[3], L[4], L[5]), c - nL,
                                                area_of(R[0], R[1], R[2], R[3], R[4], R[5]));
                    if (sc < bestCost) {
                        bestCost = sc;
                        key = split_key(sc, a, ob, tid);
                        bestN = nL;
#pragma unroll
                        for (int k = 0; k < 6; ++k) {
                            bestL[k] = L[k];
                            bestR[k] = R[k];
                        }
                    }
                }
                if (key != kNoSplit) atomicMin(&s.key[nd - ls], key);
            }
            __syncthreads();
            // the winner (or, without a candidate, the first reference) makes the leaf or the children
            if (direct) {
                const unsigned long long won = s.key[nd - ls];
                if (won == kNoSplit ? tid == b && c > (uint32_t)kMaxLeafTris : won == key) {
                    // SAH with unit traversal and intersection costs
                    const float area = s.area[nd], splitCost = __uint_as_float((uint32_t)(won >> 32));
                    if (won == kNoSplit) {
                        bestN = c / 2u;
                        median_boxes(s, b, c, bestL, bestR);
                    }
                    if (won == kNoSplit || c > (uint32_t)kMaxLeafTris ||
                        !(__fmul_rn(float(c), area) <= __fadd_rn(area, splitCost)))
                        sub_children(s, bnodes, task.node, b0, nd, bestN, bestL, bestR);
                }
            }
            __syncthreads();
            // stable partition of the split nodes' references
            const bool split = active && s.left[nd] != kNoChild;
            float4 pa, pb;
            bool lf = false;
            if (live) {
                pa = s.pa[tid];
                pb = s.pb[tid];
            }
            if (split) lf = key_left(s.key[nd - ls], __float_as_uint(pb.z), tid - b, c);
            const uint32_t bits = __ballot_sync(0xffffffffu, lf);
            if (lane_id() == 0) s.leftBits[tid >> 5] = bits;
            if (tid == 0) {
                s.levelEnd = s.nodeTop;
                s.binCount = 0;
            }
            __syncthreads();
            if (split) {
                const uint32_t ch = s.left[nd], w0 = b >> 5, w1 = tid >> 5;
                uint32_t rank = __popc(bits & ((1u << lane_id()) - 1u) & (w0 == w1 ? 0xffffffffu << (b & 31u) : 0xffffffffu));
                if (w0 != w1) rank += __popc(s.leftBits[w0] & (0xffffffffu << (b & 31u)));
                for (uint32_t w = w0 + 1; w < w1; ++w) rank += __popc(s.leftBits[w]);
                const uint32_t dst = lf ? b + rank : b + s.count[ch] + (tid - b - rank);
                s.pa[dst] = pa;
                s.pb[dst] = pb;
                s.posNode[dst] = (uint16_t)(lf ? ch : ch + 1u);
            }
            ls = le;
            le = s.levelEnd;
            ++lev;
            __syncthreads();
        }
        if (tid == 0) {
            s.levelStart[lev] = (uint16_t)ls;
            atomicMax(cnt + kCntLevels, task.level + lev);
            atomicAdd(cnt + kCntRealNodes, s.nodeTop - 1u);
        }
        if (live) order[b0 + tid] = __float_as_uint(s.pb[tid].w);
        __syncthreads();
        if (sah) {  // the cost program, deepest level first (the bins' memory now holds the costs)
            for (uint32_t l = lev; l-- > 0;) {
                for (uint32_t nd = s.levelStart[l] + tid; nd < s.levelStart[l + 1]; nd += kSubThreads) {
                    const uint32_t ch = s.left[nd], id = nd == 0 ? task.node : s.idBase + nd - 1;
                    float C[kCosts];
                    uint32_t pick = 0;
                    if (ch == kNoChild) {
                        const float leaf = leaf_cost(s.area[nd], s.count[nd], triCost);
#pragma unroll
                        for (int j = 0; j < kCosts; ++j) C[j] = leaf;
                    } else {
                        float side[2][kCosts];
#pragma unroll
                        for (uint32_t k = 0; k < 2; ++k) {
                            const uint32_t x = ch + k, xc = s.left[x];
                            const float leaf = leaf_cost(s.area[x], s.count[x], triCost);
#pragma unroll
                            for (int j = 0; j < kCosts; ++j)
                                side[k][j] = xc == kNoChild ? leaf : s.cost[((xc - 1u) >> 1) * kCosts + j];
                        }
                        pick = collapse_cost(side[0], side[1], s.area[nd], s.count[nd], triCost, C);
#pragma unroll
                        for (int j = 0; j < kCosts; ++j) s.cost[((ch - 1u) >> 1) * kCosts + j] = C[j];
                    }
                    choice[id] = pick;
                    if (nd == 0)
#pragma unroll
                        for (int j = 0; j < kCosts; ++j) cost[8ull * id + j] = C[j];
                }
                __syncthreads();
            }
        }
    }
}

AG_D float bn_area(const BinNode& b) { return area_of(b.lo.x, b.lo.y, b.lo.z, b.hi.x, b.hi.y, b.hi.z); }

// A row of the cost program: seven values in 32 bytes.
AG_D void load_costs(const float* cost, uint32_t x, float C[kCosts])
{
    const float4* row = reinterpret_cast<const float4*>(cost + 8ull * x);
    const float4 a = row[0], b = row[1];
    C[0] = a.x; C[1] = a.y; C[2] = a.z; C[3] = a.w;
    C[4] = b.x; C[5] = b.y; C[6] = b.z;
}

// One block: the cost program over the big nodes (deepest level first; a few
// round trips to L2 per level bound it: rows as 16-byte words, 34 to 25 us on
// 1M triangles, B200), then
// the collapse's start. A tree that was not finished, or is deeper than
// maxLevels, leaves the collapse without items (the previous tree stays in
// place); status (may be null) then gets kErrBuildDepth.
constexpr int kTopThreads = 1024;
__global__ void __launch_bounds__(kTopThreads) k_top(const BinNode* bnodes, float* cost,
                                                     uint32_t* choice, float triCost, bool sah,
                                                     uint2* items, uint32_t* cnt,
                                                     uint32_t levels, uint32_t maxLevels, uint32_t* status)
{
    chain_wait();
    if (cnt[kCntFailed] != 0u || cnt[kCntLevels] > maxLevels) {
        if (threadIdx.x == 0) {
            cnt[kCntFailed] |= kFailLevels;
            if (status) atomicOr(status, kErrBuildDepth);
        }
        return;
    }
    if (sah)
        for (uint32_t l = levels; l-- > 0;) {
            const uint32_t end = cnt[kLevelNodes + l + 1];
            for (uint32_t x = cnt[kLevelNodes + l] + threadIdx.x; x < end; x += kTopThreads) {
                const BinNode b = bnodes[x];
                if (b.count <= kSmallMax) continue;  // done by k_subtree
                float C[kCosts], L[kCosts], R[kCosts];
                load_costs(cost, (uint32_t)b.left, L);
                load_costs(cost, (uint32_t)b.right, R);
                choice[x] = collapse_cost(L, R, bn_area(b), b.count, triCost, C);
                float4* out = reinterpret_cast<float4*>(cost + 8ull * x);
                out[0] = make_float4(C[0], C[1], C[2], C[3]);
                out[1] = make_float4(C[4], C[5], C[6], 0.0f);
            }
            __syncthreads();
        }
    if (threadIdx.x == 0) {
        const float area = bn_area(bnodes[0]);
        cnt[kCntRootAreaInv] = __float_as_uint(area > 0.0f ? __fdiv_rn(1.0f, area) : 0.0f);
        items[0] = make_uint2(0u, 0u);
        cnt[kWideItems] = 1u;
        cnt[kWideNodeBase] = 1u;
        cnt[kWideTriBase] = 0u;
    }
}

// --------------------------------------------------------------------------
// Collapse to the wide layout: eight lanes per wide node.
constexpr int kWideThreads = 256;
constexpr uint32_t kWideItemsPerBlock = kWideThreads / 8;

// The slots of one wide node per group of eight lanes: lane g of a group
// stands for the g-th of the node's entries, left to right. choice (the cost
// program's decisions) selects the SAH-optimal distribution; null selects the
// greedy rule. The entries are then assigned to octants, and the block's
// counts kept for k_wide_emit's prefix sums. Bound by issue on the large
// levels and by the entries' loads, one after the other, on the small ones: a
// lane asks only the entry that owns it for its part of a split, and the
// octant rounds reduce values alone, with the winner found by a ballot. The
// largest level of 1M triangles: 75 to 53 us (B200).
__global__ void __launch_bounds__(kWideThreads, 8) k_wide_decide(const uint2* items,
                                                              const BinNode* bnodes,
                                                              const uint32_t* choice,
                                                              int32_t* slots, uint2* itemOff,
                                                              uint2* blockSum, uint32_t* cnt,
                                                              uint32_t level, uint32_t capItems)
{
    chain_wait();
    __shared__ uint32_t sInt[kWideItemsPerBlock], sTri[kWideItemsPerBlock], sSlots[kWideItemsPerBlock];
    const uint32_t n = min(cnt[kWideItems + level], capItems);
    const uint32_t g = threadIdx.x & 7u, gshift = lane_id() & 24u;
    constexpr uint32_t kAll = 0xffffffffu;
    for (uint32_t blk = blockIdx.x; blk * kWideItemsPerBlock < n; blk += gridDim.x) {
        const uint32_t local = threadIdx.x >> 3, i = blk * kWideItemsPerBlock + local;
        const bool valid = i < n;
        const uint32_t node = valid ? items[i].x : 0u;
        const BinNode root = bnodes[node];
        const bool single = root.count <= (uint32_t)kMaxLeafTris || root.left < 0;  // a tree of one leaf
        int32_t ent = -1;
        uint32_t count = 0;
        int32_t entLeft = -1, entRight = -1;
        auto load_entry = [&]() {
            const BinNode* b = bnodes + ent;
            const int2 lr = *reinterpret_cast<const int2*>(&b->left);
            entLeft = lr.x;
            entRight = lr.y;
            count = b->count;
        };
        if (valid && single && g == 0) ent = (int32_t)node;
        if (choice) {
            // an entry owns j consecutive lanes from its own; splitting it hands the last j - k to the right child
            uint32_t j = 1;
            if (valid && !single) {
                const uint32_t k8 = min(max(choice[node] >> 28, 1u), 7u);  // 1..7 by construction
                if (g == 0) { ent = root.left; j = k8; }
                if (g == k8) { ent = root.right; j = 8u - k8; }
            }
            bool open = ent >= 0 && j > 1u;
            while (__any_sync(kAll, open)) {
                int32_t give = -1;
                uint32_t giveSlots = 0, target = 8u;
                if (open) {
                    load_entry();
                    const uint32_t ch = choice[ent];
                    uint32_t k = 0;
                    if (entLeft >= 0)
                        while (j > 1u && (k = (ch >> (4 * (j - 1))) & 0xfu) == 0u) --j;
                    if (entLeft < 0 || j <= 1u || k == 0u || k >= j) {
                        open = false;
                    } else {
                        give = entRight;
                        giveSlots = j - k;
                        target = g + k;
                        ent = entLeft;
                        j = k;
                        open = j > 1u;
                    }
                }
                // an empty lane belongs to the nearest entry below it
                const uint32_t owners = (__ballot_sync(kAll, ent >= 0) >> gshift) & ((2u << g) - 1u);
                const int from = owners ? 31 - __clz(owners) : (int)g;
                const uint32_t t = __shfl_sync(kAll, target, from, 8), gs = __shfl_sync(kAll, giveSlots, from, 8);
                const int32_t e = __shfl_sync(kAll, give, from, 8);
                if (t == g) {
                    ent = e;
                    j = gs;
                    open = j > 1u;
                }
            }
        } else {
            // Open children until all 8 slots are used: first those too large for
            // a leaf slot, then small internal ones (tighter leaf boxes are free
            // since every slot box is tested anyway).
            uint32_t used = valid && !single ? 2u : 8u;
            float area = -1.0f;
            auto load_full = [&]() {
                load_entry();
                const float a = bn_area(bnodes[ent]);
                area = entLeft >= 0 && a >= 0.0f ? a : -1.0f;
            };
            if (valid && !single && g < 2) {
                ent = g ? root.right : root.left;
                load_full();
            }
            for (int phase = 0; phase < 2; ++phase) {
                bool active = used < 8u;
                while (__any_sync(kAll, active)) {
                    const bool large = count > (uint32_t)kMaxLeafTris;
                    float a = active && ent >= 0 && (phase == 0 ? large : !large) ? area : -1.0f;
                    uint32_t bl = g;
#pragma unroll
                    for (int o = 1; o < 8; o <<= 1) {
                        const float oa = __shfl_xor_sync(kAll, a, o, 8);
                        const uint32_t ol = __shfl_xor_sync(kAll, bl, o, 8);
                        if (oa > a || (oa == a && ol < bl)) { a = oa; bl = ol; }
                    }
                    const int32_t r = __shfl_sync(kAll, entRight, bl, 8);
                    if (!(a >= 0.0f)) active = false;
                    if (active) {
                        if (g == bl) { ent = entLeft; load_full(); }
                        if (g == used) { ent = r; load_full(); }
                        active = ++used < 8u;
                    }
                }
            }
        }
        // Octant slot assignment: slot s prefers the child whose centre lies
        // toward corner s of the parent box (bit k of s set = + side of axis k).
        float v[kWidth];
        {
            float3 cen = mk3(0.0f, 0.0f, 0.0f);
            if (ent >= 0) {
                const BinNode c = bnodes[ent];
                count = c.count;
                cen = 0.5f * (c.lo + c.hi) - 0.5f * (root.lo + root.hi);
            }
#pragma unroll
            for (int s = 0; s < kWidth; ++s)
                v[s] = ((s & 1) ? cen.x : -cen.x) + ((s & 2) ? cen.y : -cen.y) + ((s & 4) ? cen.z : -cen.z);
        }
        // The group's largest value wins its slot, the first entry and its lowest
        // slot on ties; a taken slot falls to -inf. A centre that is not a
        // number still takes a free slot, after all others.
#pragma unroll
        for (int s = 0; s < kWidth; ++s) v[s] = v[s] > -FLT_MAX ? v[s] : -FLT_MAX;
        uint32_t source = 8u;  // the entry of this lane's slot
        bool open = ent >= 0;
        while (__any_sync(kAll, open)) {
            float bv = v[0];
#pragma unroll
            for (int s = 1; s < kWidth; ++s) bv = fmaxf(bv, v[s]);
            uint32_t best = 0;
#pragma unroll
            for (int s = kWidth - 1; s >= 0; --s)
                if (v[s] == bv) best = (uint32_t)s;
            if (!open) bv = -INFINITY;
            float top = bv;
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) top = fmaxf(top, __shfl_xor_sync(kAll, top, o, 8));
            const uint32_t winners = (__ballot_sync(kAll, open && bv == top) >> gshift) & 0xffu;
            const uint32_t winner = winners ? (uint32_t)__ffs((int)winners) - 1u : 0u;
            const uint32_t slot = __shfl_sync(kAll, best, (int)winner, 8);
            if (winners) {
                if (winner == g) open = false;
                if (slot == g) source = winner;
#pragma unroll
                for (int s = 0; s < kWidth; ++s)
                    if (slot == (uint32_t)s) v[s] = -INFINITY;
            }
        }
        // from entries (by lane) to slots (by lane)
        int32_t slot = __shfl_sync(kAll, ent, (int)(source & 7u), 8);
        const uint32_t slotCount = __shfl_sync(kAll, count, (int)(source & 7u), 8);
        if (source == 8u) slot = -1;
        if (valid) slots[size_t(i) * kWidth + g] = slot;
        const bool leaf = slot >= 0 && slotCount <= (uint32_t)kMaxLeafTris;
        const uint32_t ni = __popc((__ballot_sync(kAll, slot >= 0 && !leaf) >> gshift) & 0xffu);
        const uint32_t ns = __popc((__ballot_sync(kAll, slot >= 0) >> gshift) & 0xffu);
        uint32_t nt = leaf ? slotCount : 0u;
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) nt += __shfl_xor_sync(kAll, nt, o, 8);
        if (g == 0) {
            sInt[local] = ni;
            sTri[local] = nt;
            sSlots[local] = ns;
        }
        __syncthreads();
        if (threadIdx.x < 32) {
            const uint32_t a = sInt[threadIdx.x], t = sTri[threadIdx.x], sl = sSlots[threadIdx.x];
            const uint32_t ia = scan_add(a), it = scan_add(t), is = scan_add(sl);
            const uint32_t item = blk * kWideItemsPerBlock + threadIdx.x;
            if (item < n) itemOff[item] = make_uint2(ia - a, it - t);
            if (threadIdx.x == 31) {
                blockSum[blk] = make_uint2(ia, it);
                if (ia) atomicAdd(cnt + kWideItems + level + 1, ia);
                if (it) atomicAdd(cnt + kWideTris + level, it);
                atomicAdd(cnt + kCntSlots, is);
            }
        }
        __syncthreads();  // the sums are written again for the next block of items
    }
}

// A plane word of bvh.cuh: the box [lo, hi] of one axis as offsets from the
// node's origin, rounded outwards to the top 16 bits of a float. A maximum that
// no finite word reaches (infinite, NaN, or next to FLT_MAX) gets the top half
// of +inf: with a lower half of 0 the word is +inf, with any other a NaN, which
// the traversal's minimum and maximum over the axes pass over. A minimum below
// the origin, which is 0 where a node's minimum is infinite, is stored as -inf.
constexpr uint32_t kNoBound = 0x7f800000u, kBelow16 = 0xff80u;
AG_D uint32_t plane_word(float lo, float hi, float origin)
{
    float dh = __fsub_ru(hi, origin);
    dh = dh <= 0.0f ? 0.0f : dh;
    // truncated: rounded down
    const uint32_t l16 = lo >= origin ? __float_as_uint(__fsub_rd(lo, origin)) >> 16 : kBelow16;
    const uint32_t hb = __float_as_uint(dh);
    uint32_t h16 = hb >> 16;                          // read with the lower half below it
    if (((h16 << 16) | l16) < hb) ++h16;
    return min(h16 << 16, kNoBound) | l16;
}

// Writes one wide node per group of eight lanes, a lane per slot, with its
// triangle records, dealt to the lanes evenly, and the next level's items. The
// chain order -> indices -> vertices of a record bounds it: a lane per leaf
// went through it three times, a lane per record mostly does once (build of 1M
// triangles 1,983 to 1,974 us, B200). The places of a block's items
// follow from the sums of the blocks before it, so the layout is breadth
// first and does not depend on scheduling.
__global__ void __launch_bounds__(kWideThreads) k_wide_emit(const uint2* items,
                                                            const BinNode* bnodes,
                                                            const int32_t* slots,
                                                            const uint2* itemOff,
                                                            const uint2* blockSum,
                                                            const uint32_t* order,
                                                            const float* verts,
                                                            const uint32_t* idx, uint32_t ntris,
                                                            const float4* spheres,
                                                            WideNode* nodes, TriRecord* tris,
                                                            uint2* itemsNext, uint32_t* cnt,
                                                            uint32_t level, uint32_t nodeCap, uint32_t triCap,
                                                            uint32_t* status)
{
    chain_wait();
    __shared__ __align__(16) uint8_t rec[kWideItemsPerBlock][sizeof(WideNode)];
    __shared__ uint32_t from[kWideItemsPerBlock][kWidth * kMaxLeafTris];  // of a node's records, places in `order`
    __shared__ uint32_t sums[2][kWideThreads / 32];
    __shared__ float sahSums[kWideThreads / 32];
    constexpr uint32_t kAll = 0xffffffffu;
    const uint32_t n = min(cnt[kWideItems + level], nodeCap);
    if (n == 0) return;
    const uint32_t nodeBase = cnt[kWideNodeBase + level], triBase0 = cnt[kWideTriBase + level];
    const float ria = __uint_as_float(cnt[kCntRootAreaInv]);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        cnt[kWideNodeBase + level + 1] = nodeBase + cnt[kWideItems + level + 1];
        cnt[kWideTriBase + level + 1] = triBase0 + cnt[kWideTris + level];
    }
    const uint32_t g = threadIdx.x & 7u, gshift = lane_id() & 24u, local = threadIdx.x >> 3, warp = threadIdx.x >> 5;
    uint32_t summed = 0;               // blocks of items whose sums are in the two bases
    uint32_t intBase = 0, triBase = 0;
    float sah = 0.0f;
    for (uint32_t blk = blockIdx.x; blk * kWideItemsPerBlock < n; blk += gridDim.x) {
        uint32_t a = 0, t = 0;
        for (uint32_t b = summed + threadIdx.x; b < blk; b += kWideThreads) {
            const uint2 v = blockSum[b];
            a += v.x;
            t += v.y;
        }
        a = __reduce_add_sync(kAll, a);
        t = __reduce_add_sync(kAll, t);
        if (lane_id() == 0) { sums[0][warp] = a; sums[1][warp] = t; }
        __syncthreads();
#pragma unroll
        for (int w = 0; w < kWideThreads / 32; ++w) {
            intBase += sums[0][w];
            triBase += sums[1][w];
        }
        summed = blk;
        __syncthreads();  // sums are written again
        const uint32_t i = blk * kWideItemsPerBlock + local;
        const bool valid = i < n;
        const uint2 it = valid ? items[i] : make_uint2(0u, 0u);
        const uint2 off = valid ? itemOff[i] : make_uint2(0u, 0u);
        const int32_t e = valid ? slots[size_t(i) * kWidth + g] : -1;
        const BinNode nb = bnodes[it.x];
        const float p[3] = {isinf(nb.lo.x) ? 0.0f : nb.lo.x, isinf(nb.lo.y) ? 0.0f : nb.lo.y,
                            isinf(nb.lo.z) ? 0.0f : nb.lo.z};
        BinNode c = nb;
        if (e >= 0) c = bnodes[e];
        const bool leaf = e >= 0 && c.count <= (uint32_t)kMaxLeafTris, inner = e >= 0 && !leaf;
        const uint32_t imask = (__ballot_sync(kAll, inner) >> gshift) & 0xffu;
        const uint32_t rank = __popc(imask & ((1u << g) - 1u));
        uint32_t toff = leaf ? c.count : 0u;
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            const uint32_t y = __shfl_up_sync(kAll, toff, o, 8);
            if (g >= (uint32_t)o) toff += y;
        }
        const uint32_t recs = __shfl_sync(kAll, toff, 7, 8);
        if (leaf) toff -= c.count;  // triangles of the slots before this one
        const uint32_t childBase = nodeBase + intBase + off.x, triAt = triBase0 + triBase + off.y;
        uint8_t* r = rec[local];
        uint8_t meta = 0;
        if (leaf) meta = (uint8_t)((((1u << c.count) - 1u) << 5) | toff);
        if (inner) meta = (uint8_t)(0x20u | (24u + g));
        r[24 + g] = meta;
        uint32_t* u = reinterpret_cast<uint32_t*>(r);
        // an empty slot's box is inside out: minimum 1e30, maximum -1e30
        constexpr uint32_t kEmptyPlanes = 0xf1497149u;
        const uint32_t wy = plane_word(c.lo.y, c.hi.y, p[1]), wz = plane_word(c.lo.z, c.hi.z, p[2]);
        uint32_t wx = plane_word(c.lo.x, c.hi.x, p[0]);
        // unbounded on every axis: one must not be a NaN (a minimum of -inf
        // leaves the largest finite word, 2^-17 below FLT_MAX)
        if (min(wx, min(wy, wz)) >= kNoBound) wx = (wx & 0xffffu) == kBelow16 ? 0x7f7f0000u | kBelow16 : kNoBound;
        u[8 + g] = e >= 0 ? wx : kEmptyPlanes;
        u[16 + g] = e >= 0 ? wy : kEmptyPlanes;
        u[24 + g] = e >= 0 ? wz : kEmptyPlanes;
        if (g == 0) {
            float* f = reinterpret_cast<float*>(r);
            f[0] = p[0];
            f[1] = p[1];
            f[2] = p[2];
            u[3] = imask;
            u[4] = childBase;
            u[5] = triAt;
            if (valid) sah += bn_area(nb) * ria;  // one node visit
        }
        __syncwarp();
        if (valid && g < sizeof(WideNode) / 16) {
            if (it.y < nodeCap)
                reinterpret_cast<uint4*>(nodes + it.y)[g] = reinterpret_cast<const uint4*>(r)[g];
            else
                atomicOr(status, kErrBadIndex);
        }
        __syncwarp();
        if (inner) {
            const uint32_t at = intBase + off.x + rank;
            if (at < nodeCap) itemsNext[at] = make_uint2((uint32_t)e, childBase + rank);
            else atomicOr(status, kErrBadIndex);
        }
        if (leaf) {
            sah += bn_area(c) * ria * float(c.count);
            for (uint32_t k = 0; k < c.count; ++k) from[local][toff + k] = c.begin + k;
        }
        __syncwarp();
        for (uint32_t k = g; k < recs; k += 8u) {
            const uint32_t prim = order[from[local][k]], at = triAt + k;
            TriRecord tr;
            if (prim >= ntris) {  // a sphere record
                const float4 sp = spheres[prim - ntris];
                tr.v0 = make_float4(sp.x, sp.y, sp.z, __uint_as_float(kSpherePrim | (prim - ntris)));
                tr.e0 = make_float4(fabsf(sp.w), 0.0f, 0.0f, __uint_as_float(kSphereTag));
                tr.e1 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            } else {
                const uint32_t* ti = idx + 3ull * prim;
                float v0[3], v1[3], v2[3];
#pragma unroll
                for (int x = 0; x < 3; ++x) {
                    v0[x] = verts[3ull * ti[0] + x];
                    v1[x] = verts[3ull * ti[1] + x];
                    v2[x] = verts[3ull * ti[2] + x];
                }
                tr.v0 = make_float4(v0[0], v0[1], v0[2], __uint_as_float(prim));
                tr.e0 = make_float4(__fsub_rn(v1[0], v0[0]), __fsub_rn(v1[1], v0[1]), __fsub_rn(v1[2], v0[2]), 0.0f);
                tr.e1 = make_float4(__fsub_rn(v2[0], v0[0]), __fsub_rn(v2[1], v0[1]), __fsub_rn(v2[2], v0[2]), 0.0f);
            }
            if (at < triCap) tris[at] = tr;
            else atomicOr(status, kErrBadIndex);
        }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) sah += __shfl_xor_sync(kAll, sah, o);
    if (lane_id() == 0) sahSums[warp] = sah;
    __syncthreads();
    if (threadIdx.x == 0) {
        float s = 0.0f;
        for (int w = 0; w < kWideThreads / 32; ++w) s += sahSums[w];
        if (s != 0.0f) atomicAdd(reinterpret_cast<float*>(cnt + kCntSah), s);
    }
}

// End of a device-driven build: a tree that needed more collapse levels than
// were enqueued, or is deeper than the traversal stack, is reported.
__global__ void k_end(const uint32_t* cnt, uint32_t n, uint32_t wideLevels, uint32_t* status)
{
    if (cnt[kCntFailed] != 0u) return;  // reported by k_top
    uint32_t depth = 0, tris = 0;
    for (uint32_t l = 0; l < wideLevels; ++l) {
        if (cnt[kWideItems + l] != 0u) ++depth;
        tris += cnt[kWideTris + l];
    }
    if (cnt[kWideItems + wideLevels] != 0u || depth > (uint32_t)kTraversalStack || tris != n)
        atomicOr(status, kErrBuildDepth);
}

template <typename T>
T* carve(char*& p, size_t count)
{
    size_t bytes = (count * sizeof(T) + 255) & ~size_t(255);
    T* r = reinterpret_cast<T*>(p);
    p += bytes;
    return r;
}
template <typename T>
size_t carve_bytes(size_t count)
{
    return (count * sizeof(T) + 255) & ~size_t(255);
}

inline unsigned blocks_for(size_t n, int threads, size_t cap = 0x7fffffff)
{
    const size_t b = (n + threads - 1) / threads;
    return (unsigned)(b < 1 ? 1 : (b > cap ? cap : b));
}

// A launch that may overlap the end of the kernel before it on the stream.
template <typename... P, typename... A>
void launch_chained(void (*kernel)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t st, A... args)
{
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

// Capacities of the big-task lists: at most N / (kSmallMax + 1) tasks on a
// level, and one partial chunk for each.
inline size_t max_big(size_t N) { return N / kSmallMax + 2; }
inline size_t max_chunks(size_t N) { return N / kChunk + max_big(N) + 2; }

// Halvings until at most `per` of n primitives are left: the binary depth of a
// balanced tree over them.
inline uint32_t expected_levels(uint32_t n, uint32_t per)
{
    uint32_t bits = 0;
    while (bits < 31 && (n >> bits) > per) ++bits;
    return bits;
}

}  // namespace

Builder::~Builder() { release(); }

void Builder::release()
{
    if (graphExec_) cudaGraphExecDestroy(graphExec_);
    graphExec_ = nullptr;
    graphKey_.clear();
    if (mem_) cudaFree(mem_);
    if (hostCounters_) cudaFreeHost(hostCounters_);
    if (ev0_) cudaEventDestroy(ev0_);
    if (ev1_) cudaEventDestroy(ev1_);
    mem_ = nullptr;
    hostCounters_ = nullptr;
    ev0_ = ev1_ = nullptr;
    cap_ = 0;
    bigLevels_ = wideLevels_ = 0;
}

int Builder::reserve(uint32_t n, char* err, size_t errLen)
{
    if (n <= cap_ && mem_) return 0;
    release();
    const size_t N = n ? n : 1;
    const size_t maxBig = max_big(N), maxChunks = max_chunks(N);
    char* p = nullptr;
    // the same carving twice: sizes from a null base, then the pointers
    for (int pass = 0; pass < 2; ++pass) {
        boxes_ = carve<float4>(p, 2 * N);
        for (int k = 0; k < 2; ++k) {
            refs_[k] = carve<uint32_t>(p, N);
            tasks_[k] = carve<BigTask>(p, maxBig);
            chunkTask_[k] = carve<uint32_t>(p, maxChunks);
            bins_[k] = carve<uint32_t>(p, maxBig * kTaskBinWords);
            items_[k] = reinterpret_cast<uint32_t*>(carve<uint2>(p, N + 1));
        }
        order_ = carve<uint32_t>(p, N);
        bnodes_ = carve<BinNode>(p, 2 * N);
        small_ = carve<SmallTask>(p, N);
        chunkCnt_ = carve<uint16_t>(p, maxChunks * kChunkCounts);
        chunkLeft_ = carve<uint32_t>(p, maxChunks);
        splits_ = carve<BigSplit>(p, maxBig);
        slots_ = carve<int32_t>(p, (N + 1) * kWidth);
        itemOff_ = carve<uint2>(p, N + 1);
        blockSum_ = carve<uint2>(p, (N + 1) / kWideItemsPerBlock + 1);
        collapseCost_ = carve<float>(p, 2 * N * 8);
        collapseChoice_ = carve<uint32_t>(p, 2 * N);
        counters_ = carve<uint32_t>(p, kAllWords);
        if (pass == 0) {
            const size_t bytes = (size_t)(uintptr_t)p;
            if (cudaMalloc(&mem_, bytes) != cudaSuccess) {
                snprintf(err, errLen, "BVH build: cudaMalloc of %zu bytes failed", bytes);
                mem_ = nullptr;
                cudaGetLastError();
                return -5;
            }
            p = static_cast<char*>(mem_);
        }
    }
    if (cudaMallocHost(&hostCounters_, kAllWords * sizeof(uint32_t)) != cudaSuccess) {
        snprintf(err, errLen, "BVH build: cudaMallocHost failed");
        cudaGetLastError();
        release();
        return -5;
    }
    cudaEventCreate(&ev0_);
    cudaEventCreate(&ev1_);
    cap_ = n;
    return 0;
}

void Builder::launch_begin(const Input& in, cudaStream_t st)
{
    const uint32_t n = in.ntris + in.nspheres;
    k_begin<<<4, 1024, 0, st>>>(counters_);
    launch_chained(k_prep_prims, blocks_for(n, kPrepThreads, 148 * 8), kPrepThreads, 0, st, in.verts, in.idx, in.ntris,
                   in.spheres, n, boxes_, refs_[0], counters_ + kCntBounds);
    const size_t rootThreads = std::max<size_t>(n > kSmallMax ? (n + kChunk - 1) / kChunk : 1, kTaskBinWords);
    launch_chained(k_root, blocks_for(rootThreads, 256), 256, 0, st, n, counters_, static_cast<BigTask*>(tasks_[0]),
                   bnodes_, static_cast<SmallTask*>(small_), chunkTask_[0], bins_[0]);
}

// Binary levels [first, last) of the big tasks.
void Builder::launch_big_levels(const Input& in, uint32_t first, uint32_t last, cudaStream_t st)
{
    const uint32_t n = in.ntris + in.nspheres;
    const uint32_t capBig = (uint32_t)max_big(n), capChunks = (uint32_t)max_chunks(n);
    BigSplit* splits = static_cast<BigSplit*>(splits_);
    for (uint32_t L = first; L < last; ++L) {
        const int a = L & 1u, b = a ^ 1;
        BigTask *cur = static_cast<BigTask*>(tasks_[a]), *next = static_cast<BigTask*>(tasks_[b]);
        // level L has at most 2^L tasks; the kernels loop, so any grid covers them
        const size_t tasks = std::min<size_t>(L < 20 ? size_t(1) << L : capBig, n / (kSmallMax + 1) + 1);
        const unsigned gTasks = blocks_for(tasks, 1, 148 * 8), gChunks = blocks_for(n / kChunk + tasks, 1, 148 * 8);
        launch_chained(k_bin, gChunks, kChunkThreads, 0, st, cur, refs_[a], boxes_, chunkTask_[a], bins_[a], chunkCnt_,
                       counters_, L, capChunks);
        launch_chained(k_split, gTasks, kSplitThreads, 0, st, cur, bins_[a], chunkCnt_, chunkLeft_, splits, bnodes_,
                       next, chunkTask_[b], bins_[b], static_cast<SmallTask*>(small_), counters_, L, capBig, capChunks,
                       n, in.status);
        launch_chained(k_scatter, gChunks, kChunkThreads, 0, st, next, cur, refs_[a], refs_[b], boxes_, chunkTask_[a],
                       splits, chunkLeft_, counters_, L, capChunks, in.status);
    }
}

// The subtrees, the top of the cost program and the collapse's start.
void Builder::launch_subtrees(const Input& in, uint32_t levels, uint32_t maxLevels, bool report, cudaStream_t st)
{
    const uint32_t n = in.ntris + in.nspheres;
    const bool sah = collapse_ == kCollapseSah;
    cudaFuncSetAttribute(k_subtree, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SubSmem));
    launch_chained(k_subtree, blocks_for(n, 64, 148 * 2), kSubThreads, sizeof(SubSmem), st,
                   static_cast<const SmallTask*>(small_), refs_[0], refs_[1], boxes_, bnodes_, order_, collapseCost_,
                   collapseChoice_, triCost_, sah, counters_, levels, n);
    launch_chained(k_top, 1, kTopThreads, 0, st, bnodes_, collapseCost_, collapseChoice_, triCost_, sah,
                   reinterpret_cast<uint2*>(items_[0]), counters_, levels, maxLevels, report ? in.status : nullptr);
}

// Collapse levels [first, last).
void Builder::launch_wide_levels(const Input& in, uint32_t first, uint32_t last, cudaStream_t st)
{
    const uint32_t n = in.ntris + in.nspheres;
    uint2 *off = static_cast<uint2*>(itemOff_), *sums = static_cast<uint2*>(blockSum_);
    for (uint32_t D = first; D < last; ++D) {
        uint2 *cur = reinterpret_cast<uint2*>(items_[D & 1u]), *next = reinterpret_cast<uint2*>(items_[(D & 1u) ^ 1u]);
        // level D has at most 8^D wide nodes
        const size_t items = std::min<size_t>(D < 7 ? size_t(1) << (3 * D) : n + 1, n + 1);
        const unsigned grid = blocks_for(items, (int)kWideItemsPerBlock, 148 * 8);
        launch_chained(k_wide_decide, grid, kWideThreads, 0, st, cur, bnodes_,
                       collapse_ == kCollapseSah ? collapseChoice_ : nullptr, slots_, off, sums, counters_, D, n + 1);
        launch_chained(k_wide_emit, grid, kWideThreads, 0, st, cur, bnodes_, slots_, off, sums, order_, in.verts, in.idx,
                       in.ntris, in.spheres, in.nodes, in.tris, next, counters_, D, n + 1, n, in.status);
    }
}

// Statistics from the counter words of a finished build.
BuildStats Builder::stats_of(const uint32_t* h) const
{
    BuildStats s;
    s.binaryNodes = h[kCntRealNodes];
    s.binaryLevels = h[kCntLevels];
    for (uint32_t L = 0; L < kMaxLevels && h[kLevelBig + L]; ++L) s.bigLevels = L + 1;
    for (uint32_t D = 0; D <= kMaxWideLevels; ++D) {
        s.wideNodes += h[kWideItems + D];
        s.triCount += h[kWideTris + D];
        if (h[kWideItems + D]) s.wideDepth = D + 1;
    }
    s.sahCost = __builtin_bit_cast(float, h[kCntSah]);
    s.childSlots = h[kCntSlots];
    return s;
}

int Builder::build(const float* verts, const uint32_t* idx, uint32_t ntris, const float4* spheres, uint32_t nspheres,
                   WideNode* nodes, TriRecord* tris, uint32_t* deviceStatus, cudaStream_t st, BuildStats* stats,
                   char* err, size_t errLen)
{
    const uint32_t n = ntris + nspheres;
    BuildStats local;
    if (n == 0) {
        if (stats) *stats = local;
        return 0;
    }
    if (int rc = reserve(n, err, errLen)) return rc;
    const Input in{verts, idx, ntris, spheres, nspheres, nodes, tris, deviceStatus};
    // levels enqueued at first: the last build's and one more, or those of a
    // balanced tree (three binary levels to a collapse level) with a margin of 3
    // and 4 for uneven ones. A big level without tasks costs three empty
    // launches, a collapse level without items two; one too few costs a wait.
    uint32_t levels = n > kSmallMax ? (bigLevels_ ? bigLevels_ + 1u : expected_levels(n, kSmallMax) + 3u) : 0u;
    uint32_t wide = wideLevels_ ? wideLevels_ + 1u : 4u + expected_levels(n, 1) / 3u;
    levels = std::min(levels, kMaxLevels);
    wide = std::min(wide, kMaxWideLevels);
    uint32_t* h = hostCounters_;
    auto read_counters = [&]() -> int {
        cudaEventRecord(ev1_, st);
        cudaMemcpyAsync(h, counters_, kAllWords * sizeof(uint32_t), cudaMemcpyDeviceToHost, st);
        if (cudaStreamSynchronize(st) == cudaSuccess) return 0;
        snprintf(err, errLen, "BVH build: %s", cudaGetErrorString(cudaGetLastError()));
        return -2;
    };
    cudaEventRecord(ev0_, st);
    launch_begin(in, st);
    launch_big_levels(in, 0, levels, st);
    launch_subtrees(in, levels, kMaxLevels, false, st);
    launch_wide_levels(in, 0, wide, st);
    if (int rc = read_counters()) return rc;
    while (h[kLevelBig + levels] != 0u && !(h[kCntFailed] & kFailCapacity)) {  // big tasks below the levels enqueued: nothing after them has run
        if (levels >= kMaxLevels) {
            snprintf(err, errLen, "BVH build: more than %u levels", kMaxLevels);
            return -4;
        }
        const uint32_t more = std::min(kMaxLevels, levels + std::max(8u, levels / 2));
        cudaMemsetAsync(counters_ + kCntFailed, 0, sizeof(uint32_t), st);
        launch_big_levels(in, levels, more, st);
        levels = more;
        launch_subtrees(in, levels, kMaxLevels, false, st);
        launch_wide_levels(in, 0, wide, st);
        if (int rc = read_counters()) return rc;
    }
    if (h[kCntLevels] > kMaxLevels) {
        snprintf(err, errLen, "BVH build: more than %u levels", kMaxLevels);
        return -4;
    }
    while (h[kWideItems + wide] != 0u) {
        if (wide >= kMaxWideLevels) {
            snprintf(err, errLen, "BVH collapse: more than %u wide levels", kMaxWideLevels);
            return -4;
        }
        const uint32_t more = std::min(kMaxWideLevels, wide + 8u);
        launch_wide_levels(in, wide, more, st);
        wide = more;
        if (int rc = read_counters()) return rc;
    }
    local = stats_of(h);
    bigLevels_ = local.bigLevels;
    wideLevels_ = local.wideDepth;
    cudaEventElapsedTime(&local.buildMs, ev0_, ev1_);
    if (h[kCntFailed] != 0u || local.triCount != n) {
        snprintf(err, errLen, "BVH build: %u primitives placed, expected %u", local.triCount, n);
        return -3;
    }
    if (local.wideDepth > (uint32_t)kTraversalStack) {
        snprintf(err, errLen, "BVH build: wide depth %u exceeds the traversal stack (%d)", local.wideDepth,
                 kTraversalStack);
        return -4;
    }
    if (stats) *stats = local;
    return 0;
}

void Builder::enqueue_launches(const Input& in, uint32_t maxLevels, uint32_t maxWideLevels, cudaStream_t st)
{
    const uint32_t n = in.ntris + in.nspheres;
    // tasks above kSmallMax references occur on the top levels only: their
    // kernels run on the levels where the last build() had them, plus a margin
    // (k_subtree reports a big task left after them)
    const uint32_t levels = n > kSmallMax ? std::min(maxLevels, bigLevels_ + 2u) : 0u;
    launch_begin(in, st);
    launch_big_levels(in, 0, levels, st);
    launch_subtrees(in, levels, maxLevels, true, st);
    launch_wide_levels(in, 0, maxWideLevels, st);
    k_end<<<1, 1, 0, st>>>(counters_, n, maxWideLevels, in.status);
}

int Builder::enqueue(const float* verts, const uint32_t* idx, uint32_t ntris, const float4* spheres,
                     uint32_t nspheres, WideNode* nodes, TriRecord* tris, uint32_t* deviceStatus, cudaStream_t st,
                     uint32_t maxLevels, uint32_t maxWideLevels, char* err, size_t errLen)
{
    const uint32_t n = ntris + nspheres;
    if (n == 0) return 0;
    if (!mem_ || n > cap_) {
        snprintf(err, errLen, "BVH enqueue: no buffers for %u primitives (run a build of this size first)", n);
        return -6;
    }
    if (maxLevels == 0 || maxLevels > kMaxLevels || maxWideLevels == 0 || maxWideLevels > kMaxWideLevels) {
        snprintf(err, errLen, "BVH enqueue: level caps must be 1-%u (binary) and 1-%u (wide)", kMaxLevels, kMaxWideLevels);
        return -6;
    }
    const uint64_t key[] = {(uint64_t)(uintptr_t)verts, (uint64_t)(uintptr_t)idx, (uint64_t)(uintptr_t)spheres,
                            (uint64_t)(uintptr_t)nodes, (uint64_t)(uintptr_t)tris, (uint64_t)(uintptr_t)deviceStatus,
                            (uint64_t)(uintptr_t)mem_, ntris, nspheres, maxLevels, maxWideLevels, bigLevels_, collapse_,
                            (uint64_t)__builtin_bit_cast(uint32_t, triCost_)};
    const std::vector<uint64_t> k(key, key + sizeof key / sizeof key[0]);
    if (!graphExec_ || k != graphKey_) {
        if (graphExec_) cudaGraphExecDestroy(graphExec_);
        graphExec_ = nullptr;
        if (cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
            snprintf(err, errLen, "BVH enqueue: stream capture could not begin: %s",
                     cudaGetErrorString(cudaGetLastError()));
            return -2;
        }
        enqueue_launches(Input{verts, idx, ntris, spheres, nspheres, nodes, tris, deviceStatus}, maxLevels, maxWideLevels,
                         st);
        cudaGraph_t g = nullptr;
        cudaError_t e = cudaStreamEndCapture(st, &g);
        if (e == cudaSuccess) e = cudaGraphInstantiate(&graphExec_, g, 0);
        if (g) cudaGraphDestroy(g);
        if (e != cudaSuccess) {
            graphExec_ = nullptr;
            cudaGetLastError();
            snprintf(err, errLen, "BVH enqueue: graph capture: %s", cudaGetErrorString(e));
            return -2;
        }
        graphKey_ = k;
        ++graphCaptures_;
    }
    cudaEventRecord(ev0_, st);
    cudaError_t e = cudaGraphLaunch(graphExec_, st);
    cudaEventRecord(ev1_, st);
    if (e != cudaSuccess) {
        snprintf(err, errLen, "BVH enqueue: graph launch: %s", cudaGetErrorString(e));
        return -2;
    }
    ++graphLaunches_;
    return 0;
}

int Builder::enqueued_stats(cudaStream_t st, BuildStats* stats, char* err, size_t errLen)
{
    if (!mem_ || graphLaunches_ == 0) {
        snprintf(err, errLen, "BVH stats: no device-driven build yet");
        return -6;
    }
    cudaMemcpyAsync(hostCounters_, counters_, kAllWords * sizeof(uint32_t), cudaMemcpyDeviceToHost, st);
    if (cudaStreamSynchronize(st) != cudaSuccess) {
        snprintf(err, errLen, "BVH stats: %s", cudaGetErrorString(cudaGetLastError()));
        return -2;
    }
    *stats = stats_of(hostCounters_);
    float ms = 0.0f;
    if (graphLaunches_ && cudaEventElapsedTime(&ms, ev0_, ev1_) == cudaSuccess) stats->buildMs = ms;
    cudaGetLastError();
    return 0;
}

}  // namespace ag
