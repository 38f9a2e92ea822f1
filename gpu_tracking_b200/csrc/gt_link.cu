// gt_link.cu — trackpy-style optimal subnet linking on the GPU.
//
// Replaces Linker / link / recurse / recurse2 (src/linking.rs:345-816) and
// the kd-tree neighbour search (within_radius_rd2, src/linking.rs:211-247).
//
//   link_cells_kernel    points of every frame group in cells of at least the
//                        search radius (the neighbour index; the exact
//                        within_radius_rd2 predicate decides).
//   sort_groups_kernel   the index of callers without scratch: points sorted
//                        by row, bisected.
//   count/fill_lists     for every point and every lag k = 1..memory+1, the
//                        forward (dests in group+k) and backward (sources in
//                        group-k) neighbour lists in ascending point order; all
//                        frame pairs in parallel.
//   link_frames          the frame loop: one CTA walks frames in order doing
//                        each frame's work in parallel: memory merge, subnet
//                        detection by union-find, the reference's DFS order
//                        per subnet, the exact branch-and-bound per subnet
//                        (one thread each, same float operation sequence),
//                        new ids in destination order, memory ring and
//                        duration bookkeeping.
//   link_segments_kernel the loop over segments of a video's frames, one CTA
//                        each, joined where their states agree.
//   link_video_kernel    the loop over a whole video or window in one CTA:
//                        videos with linker resets, memory above 16, videos of
//                        one segment and callers without scratch.
#include "gt_kernels.h"

namespace gt {

constexpr int kLinkThreads = 1024;
constexpr int kSortSmem = 4096;
constexpr long long kSubnetBudget = 1ll << 28;
constexpr int kLagRegs = 4;     // backward-list offsets of up to 4 lags held in registers
constexpr int kEdgeRegs = 2;    // backward edges per lag gathered in registers before they are written
constexpr int kRingSmem = 64;   // memory ring bookkeeping in shared memory up to memory = 64
// A frame with at most LinkSmem<SF>::D detections and LinkSmem<SF>::S sources
// keeps its per-destination and per-source working arrays in shared memory;
// larger frames use the same arrays in the global scratch.  SF is the type of
// the per-source forward-list offsets: int32 when every offset of the lists
// fits (a larger working set in the same shared memory), int64 otherwise.
template <typename SF>
struct LinkSmem;
template <>
struct LinkSmem<int64_t> {
    static constexpr int D = 2048, S = 2560;
};
template <>
struct LinkSmem<int32_t> {
    static constexpr int D = 3840, S = 4608;
};
template <typename SF>
constexpr size_t link_smem_bytes() {
    return (size_t)(LinkSmem<SF>::D + 1) * 4 * 10 + (size_t)LinkSmem<SF>::S * (2 * sizeof(SF) + 4 + 1);
}
static_assert(((LinkSmem<int64_t>::D + 1) * 4 * 10) % 8 == 0, "source block stays 8-byte aligned");
static_assert(link_smem_bytes<int32_t>() + 4096 <= 227 * 1024, "the int32 working set fits with the static arrays");

// ------------------------------------------------------- point addressing
__device__ __forceinline__ int64_t gbase(const LinkInput& in, int g) {
    return in.slot_stride ? (int64_t)g * in.slot_stride : in.goff[g];
}
__device__ __forceinline__ int64_t gsize(const LinkInput& in, int g) {
    return in.slot_stride ? (int64_t)in.gcount[g] : in.goff[g + 1] - in.goff[g];
}
__device__ __forceinline__ int ggroup(const LinkInput& in, int64_t p) {
    return in.slot_stride ? (int)(p / in.slot_stride) : in.pgroup[p];
}
__device__ __forceinline__ float prow(const LinkInput& in, int64_t p) { return in.px[p * in.xy_stride]; }
__device__ __forceinline__ float pcol(const LinkInput& in, int64_t p) { return in.py[p * in.xy_stride]; }
// offset-array index of (point p, lag slot k) in 0..K
__device__ __forceinline__ int64_t lix(const LinkLists& L, int64_t p, int K, int k) {
    return (p - L.pbase) * K + k;
}

// ------------------------------------------------------------ group sorting
__global__ void __launch_bounds__(kLinkThreads)
sort_groups_kernel(LinkInput in, uint32_t* __restrict__ srt, uint64_t* __restrict__ scratch, size_t per_group) {
    __shared__ uint64_t sk[kSortSmem];
    const int g = blockIdx.x;
    const int64_t a = gbase(in, g), n = gsize(in, g);
    if (n == 0) return;
    int np2 = 1;
    while (np2 < n) np2 <<= 1;
    uint64_t* keys = (np2 <= kSortSmem) ? sk : scratch + (size_t)blockIdx.x * per_group;
    for (int i = threadIdx.x; i < np2; i += blockDim.x)
        keys[i] = (i < n) ? (((uint64_t)float_order_key(prow(in, a + i)) << 32) | (uint64_t)i) : ~0ull;
    __syncthreads();
    block_sort_u64(keys, np2);
    for (int i = threadIdx.x; i < n; i += blockDim.x) srt[a + i] = (uint32_t)(keys[i] & 0xFFFFFFFFull);
}

// -------------------------------------------------------------- cell index
// The points of a group in cells of one to sixteen search radii, side x side
// of them, which cover the group's own bounding box or, where that is larger,
// repeat over the plane: a search reads the points of the cells that its box
// touches, a handful, as (row, column, index) records.  Sorted rows alone leave
// every point of three radii of rows, a few tens, behind an index each, and a
// bisection or a row index before them.  Lists of 400 frames of 2000 points,
// memory 3: 1140 -> 260 us, and 70 -> 28 us to build the index (B200).  Cells
// that always cover the box save 5 % of that, but a few points far away gather
// all others in one cell: 50 frames of 10,000 points, one of them at 1e6, link
// in 32 ms so, 3.8 with cells that repeat, 12 with sorted rows.

// Cells a side for n points: about four a point up to 64 x 64.
__host__ __device__ inline int link_cell_side(int64_t n) {
    int s = n > 1024 ? 64 : (int)sqrtf(4.0f * (float)n);
    return s < 1 ? 1 : (s > 64 ? 64 : s);
}
// where group g's cell offsets start: side * side + 1 <= 4 n + 1 entries
__device__ __forceinline__ int64_t cell_base(const LinkInput& in, int g) {
    return in.slot_stride ? (int64_t)g * (link_cells_per_slot(in.slot_stride) + 1) : 4 * in.goff[g] + g;
}
// cell coordinate along one axis, monotone in the position (NaN: 0), and where
// it lies among the cells of a side
constexpr int kCellMax = 1 << 30;
__device__ __forceinline__ int cell_of(float v, float v0, float inv) {
    const float t = __fmul_rn(__fsub_rn(v, v0), inv);
    return t >= (float)kCellMax ? kCellMax : (t > 0.0f ? (int)t : 0);
}
__device__ __forceinline__ int cell_in(int c, int side) { return c < side ? c : c % side; }
// width of the cells over an extent
__device__ __forceinline__ float cell_width(float radius, float extent, int side) {
    const float w = fmaxf(radius, extent / (float)side);
    return radius > 0.0f ? fminf(w, 16.0f * radius) : w;
}

constexpr int kCellThreads = 512;
__global__ void __launch_bounds__(kCellThreads)
link_cells_kernel(LinkInput in, int g0, float4* __restrict__ rec, int32_t* __restrict__ cell_off,
                  float4* __restrict__ geo) {
    __shared__ int cnt[64 * 64];
    __shared__ float red[4][kCellThreads / 32];
    __shared__ int wsum[33];
    const int g = g0 + blockIdx.x, tid = threadIdx.x;
    const int64_t a = gbase(in, g), n = gsize(in, g);
    const int side = link_cell_side(n), ncell = side * side;
    int32_t* const off = cell_off + cell_base(in, g);
    float r0 = INFINITY, r1 = -INFINITY, c0 = INFINITY, c1 = -INFINITY;
    for (int64_t i = tid; i < n; i += blockDim.x) {
        const float r = prow(in, a + i), c = pcol(in, a + i);
        if (fabsf(r) < INFINITY) {
            r0 = fminf(r0, r);
            r1 = fmaxf(r1, r);
        }
        if (fabsf(c) < INFINITY) {
            c0 = fminf(c0, c);
            c1 = fmaxf(c1, c);
        }
    }
    for (int d = 16; d; d >>= 1) {
        r0 = fminf(r0, __shfl_xor_sync(0xffffffffu, r0, d));
        r1 = fmaxf(r1, __shfl_xor_sync(0xffffffffu, r1, d));
        c0 = fminf(c0, __shfl_xor_sync(0xffffffffu, c0, d));
        c1 = fmaxf(c1, __shfl_xor_sync(0xffffffffu, c1, d));
    }
    if ((tid & 31) == 0) {
        red[0][tid >> 5] = r0;
        red[1][tid >> 5] = r1;
        red[2][tid >> 5] = c0;
        red[3][tid >> 5] = c1;
    }
    for (int i = tid; i < ncell; i += blockDim.x) cnt[i] = 0;
    __syncthreads();
    for (int w = 0; w < kCellThreads / 32; w++) {
        r0 = fminf(r0, red[0][w]);
        r1 = fmaxf(r1, red[1][w]);
        c0 = fminf(c0, red[2][w]);
        c1 = fmaxf(c1, red[3][w]);
    }
    // an extent without a finite width is one cell
    float ir = 1.0f / cell_width(in.radius, r1 - r0, side), ic = 1.0f / cell_width(in.radius, c1 - c0, side);
    if (!(ir > 0.0f && ir < INFINITY)) ir = 0.0f;
    if (!(ic > 0.0f && ic < INFINITY)) ic = 0.0f;
    if (tid == 0) geo[g] = make_float4(r0, c0, ir, ic);
    auto cell = [&](float r, float c) {
        return cell_in(cell_of(r, r0, ir), side) * side + cell_in(cell_of(c, c0, ic), side);
    };
    for (int64_t i = tid; i < n; i += blockDim.x) atomicAdd(cnt + cell(prow(in, a + i), pcol(in, a + i)), 1);
    __syncthreads();
    {
        // exclusive scan, a run of 8 cells a thread
        static_assert(64 * 64 == 8 * kCellThreads, "eight cells a thread");
        int v[8], s = 0;
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const int e = tid * 8 + k;
            v[k] = e < ncell ? cnt[e] : 0;
            s += v[k];
        }
        int tot;
        int x = block_excl_scan(s, &tot, wsum);
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const int e = tid * 8 + k;
            if (e < ncell) {
                off[e] = x;
                cnt[e] = x;
            }
            x += v[k];
        }
        if (tid == 0) off[ncell] = tot;
    }
    __syncthreads();
    // (the order inside a cell does not matter: the lists are sorted)
    for (int64_t i = tid; i < n; i += blockDim.x) {
        const float r = prow(in, a + i), c = pcol(in, a + i);
        const int p = atomicAdd(cnt + cell(r, c), 1);
        rec[a + p] = make_float4(r, c, __int_as_float((int)i), 0.0f);
    }
}

// Sorted positions [p0, p1) of group t that hold every row in [lo, hi]: the
// first position whose row key is >= klo and the first > khi.
__device__ __forceinline__ void row_range(const LinkInput& in, const LinkLists& L, int t, float lo, float hi,
                                          int64_t* p0, int64_t* p1) {
    const uint32_t* srt = L.srt;
    const int64_t a = gbase(in, t), n = gsize(in, t);
    const uint32_t klo = float_order_key(lo), khi = float_order_key(hi);
    int64_t x = 0, y = n;
    while (x < y) {
        int64_t m = (x + y) >> 1;
        if (float_order_key(prow(in, a + srt[a + m])) < klo) x = m + 1; else y = m;
    }
    *p0 = x;
    y = n;
    while (x < y) {
        int64_t m = (x + y) >> 1;
        if (float_order_key(prow(in, a + srt[a + m])) <= khi) x = m + 1; else y = m;
    }
    *p1 = x;
}

__device__ __forceinline__ void search_bounds(float q, float R, float* lo, float* hi) {
    // conservative superset of the rows within_rd2 can accept
    float delta = __fmul_rn(fmaxf(fabsf(q), R), 1.0f / 1048576.0f) + 1e-30f;
    *lo = __fsub_rn(__fsub_rn(q, R), delta);
    *hi = __fadd_rn(__fadd_rn(q, R), delta);
}

// f(index, row, column) for every point of group t that within_rd2 can accept
// for a query at (qx, qy), and a few more.
template <typename F>
__device__ __forceinline__ void near_points(const LinkInput& in, const LinkLists& L, int t, float qx, float qy, F&& f) {
    float lo, hi;
    search_bounds(qx, in.radius, &lo, &hi);
    const int64_t a = gbase(in, t);
    if (L.rec) {
        const int side = link_cell_side(gsize(in, t));
        const float4 ge = L.geo[t];
        // the cells of the box, each once: runs of a side's cells that start
        // again at its first one
        int y = cell_of(lo, ge.x, ge.z);
        int rows = min(cell_of(hi, ge.x, ge.z) - y + 1, side);
        search_bounds(qy, in.radius, &lo, &hi);
        int x0 = cell_of(lo, ge.y, ge.w);
        const int cols = min(cell_of(hi, ge.y, ge.w) - x0 + 1, side);
        y = cell_in(y, side);
        x0 = cell_in(x0, side);
        const int32_t* const off = L.cell_off + cell_base(in, t);
        for (; rows > 0; rows--) {
            const int32_t* const row = off + y * side;
            for (int x = x0, left = cols; left > 0; x = 0) {
                const int run = min(left, side - x);
                for (int m = row[x], e = row[x + run]; m < e; m++) {
                    const float4 q = L.rec[a + m];
                    f(__float_as_int(q.z), q.x, q.y);
                }
                left -= run;
            }
            if (++y == side) y = 0;
        }
        return;
    }
    int64_t s0, s1;
    row_range(in, L, t, lo, hi, &s0, &s1);
    for (int64_t m = s0; m < s1; m++) {
        const int i = (int)L.srt[a + m];
        f(i, prow(in, a + i), pcol(in, a + i));
    }
}

__device__ __forceinline__ void group_video_range(const LinkInput& in, int h, int* vb, int* ve) {
    int x = 0, y = in.nvideos;  // last video with vgrp[v] <= h
    while (y - x > 1) {
        int m = (x + y) >> 1;
        if (in.vgrp[m] <= h) x = m; else y = m;
    }
    *vb = in.vgrp[x];
    *ve = in.vgrp[x + 1];
}

// mode 0: count, mode 1: fill (and sort ascending); points [p0, p1), offsets
// relative to L.pbase.  A fill whose list would pass the end of its buffer
// (f_cap / b_cap) writes nothing and raises kFlagListOverflow.
template <int kMode>
__global__ void lists_kernel(LinkInput in, LinkLists L, int64_t* f_cnt, int64_t* b_cnt, int64_t p0, int64_t p1,
                             uint32_t* flags) {
    const int64_t p = p0 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= p1) return;
    const int K = in.memory + 1;
    const int h = ggroup(in, p);
    if (in.slot_stride && p - gbase(in, h) >= gsize(in, h)) return;  // empty slot
    int vb, ve;
    group_video_range(in, h, &vb, &ve);
    const int ready = in.groups_ready > 0 ? in.groups_ready : in.ngroups;
    const float qx = prow(in, p), qy = pcol(in, p);
    const float R = in.radius;
    const bool qnan = (qx != qx) || (qy != qy);
    for (int k = 1; k <= K; k++) {
        // forward: p is a source, dests in group h + k
        int t = h + k;
        int64_t cnt = 0;
        bool skip = false;
        if (kMode && t < ve && t < ready && L.f_cap >= 0 && L.f_off[lix(L, p, K, k)] > L.f_cap) {
            atomicOr(flags, kFlagListOverflow);
            skip = true;
        }
        if (t < ve && t < ready && !qnan && !skip) {
            int32_t* out = kMode ? L.f_pts + L.f_off[lix(L, p, K, k - 1)] : nullptr;
            near_points(in, L, t, qx, qy, [&](int i, float row, float col) {
                float dist;
                if (within_rd2(row, col, qx, qy, R, &dist)) {
                    if (kMode) out[cnt] = i;
                    cnt++;
                }
            });
            if (kMode) {  // ascending destination order
                for (int64_t i = 1; i < cnt; i++) {
                    int32_t v = out[i];
                    int64_t j = i - 1;
                    while (j >= 0 && out[j] > v) { out[j + 1] = out[j]; j--; }
                    out[j + 1] = v;
                }
            }
        }
        if (!kMode) f_cnt[lix(L, p, K, k - 1)] = cnt;
        // backward: p is a dest, sources in group h - k
        t = h - k;
        cnt = 0;
        skip = false;
        if (kMode && t >= vb && L.b_cap >= 0 && L.b_off[lix(L, p, K, k)] > L.b_cap) {
            atomicOr(flags, kFlagListOverflow);
            skip = true;
        }
        if (t >= vb && !qnan && !skip) {
            int32_t* out = kMode ? L.b_pts + L.b_off[lix(L, p, K, k - 1)] : nullptr;
            float* outd = kMode ? L.b_dist + L.b_off[lix(L, p, K, k - 1)] : nullptr;
            near_points(in, L, t, qx, qy, [&](int i, float row, float col) {
                float dist;
                if (within_rd2(qx, qy, row, col, R, &dist)) {
                    if (kMode) {
                        out[cnt] = i;
                        outd[cnt] = dist;
                    }
                    cnt++;
                }
            });
            if (kMode) {  // ascending source order
                for (int64_t i = 1; i < cnt; i++) {
                    int32_t v = out[i];
                    float vd = outd[i];
                    int64_t j = i - 1;
                    while (j >= 0 && out[j] > v) { out[j + 1] = out[j]; outd[j + 1] = outd[j]; j--; }
                    out[j + 1] = v;
                    outd[j + 1] = vd;
                }
            }
        }
        if (!kMode) b_cnt[lix(L, p, K, k - 1)] = cnt;
    }
}

// ---------------------------------------------------------- scratch layout
// dblk: 10 per-destination int32 arrays of G + 1 entries (d_off, d_end,
// out_src, parent, comp_nd, comp_ns, comp_off, comp_soff, roots, tmp);
// sblk: per-source sf0, sf1 (int64), src_pt (int32), srcUsed (u8), Smax each.
struct Lay {
    size_t pids, snap, start, idstamp, firstpos, srcidx, srcstamp, ring_pt, ring_n, ringpre, dblk, sblk, e_src, e_dist, pathD,
        pathS, srcLocal, vis_d, vis_s, stack, r2a, r2b, r2c, r2used, total;
};

__host__ __device__ inline size_t al(size_t x) { return (x + 15) & ~(size_t)15; }

__host__ __device__ inline Lay make_lay(int64_t G, int64_t E, int64_t NP, int64_t M, bool spec) {
    Lay l;
    const int64_t Smax = G * (M + 1);
    size_t o = 0;
    l.start = o; o = al(o + 8 * NP);
    l.idstamp = o; o = al(o + 4 * NP);
    l.firstpos = o; o = al(o + 8 * NP);
    l.srcidx = o; o = al(o + 4 * NP);
    l.srcstamp = o; o = al(o + 4 * NP);
    l.ring_pt = o; o = al(o + 4 * (M * G + 1));
    l.ring_n = o; o = al(o + 4 * (M + 1));
    l.ringpre = o; o = al(o + 4 * (M + 2));
    l.dblk = o; o = al(o + 4 * 10 * (G + 1));
    l.sblk = o; o = al(o + (8 + 8 + 4 + 1) * Smax);
    l.e_src = o; o = al(o + 4 * (E + 1));
    l.e_dist = o; o = al(o + 4 * (E + 1));
    l.pathD = o; o = al(o + 4 * G);
    l.pathS = o; o = al(o + 4 * Smax);
    l.srcLocal = o; o = al(o + 4 * Smax);
    l.vis_d = o; o = al(o + 4 * G);
    l.vis_s = o; o = al(o + 4 * Smax);
    l.stack = o; o = al(o + 8 * (G + Smax));
    l.r2a = o; o = al(o + 4 * G);
    l.r2b = o; o = al(o + 4 * G);
    l.r2c = o; o = al(o + 4 * G);
    l.r2used = o; o = al(o + Smax);
    // speculative runs: ids of the frames before their own, ring and ring sizes as they reach them
    l.pids = o; o = spec ? al(o + 8 * NP) : o;
    l.snap = o; o = spec ? al(o + 4 * (M * G + M + 1)) : o;
    l.total = o;
    return l;
}

size_t link_scratch_bytes(int32_t max_group, int64_t max_edges, int64_t npoints_video, int32_t memory) {
    return make_lay(max_group, max_edges, npoints_video, memory, false).total;
}

void link_scratch_point_arrays(int32_t max_group, int64_t max_edges, int64_t npoints_video, int32_t memory,
                               size_t* idstamp, size_t* srcstamp, size_t* firstpos) {
    const Lay l = make_lay(max_group, max_edges, npoints_video, memory, false);
    *idstamp = l.idstamp;
    *srcstamp = l.srcstamp;
    *firstpos = l.firstpos;
}

// union-find over the destinations of one frame; roots are minimal indices
__device__ __forceinline__ int uf_find(volatile int* parent, int x) {
    while (true) {
        int p = parent[x];
        if (p == x) return x;
        int gp = parent[p];
        if (gp != p) parent[x] = gp;
        x = p;
    }
}
__device__ __forceinline__ void uf_union(volatile int* parent, int a, int b) {
    while (true) {
        a = uf_find(parent, a);
        b = uf_find(parent, b);
        if (a == b) return;
        if (a > b) { int t = a; a = b; b = t; }
        int old = atomicCAS((int*)&parent[b], b, a);
        if (old == b) return;
    }
}

// Block-wide state of a linker run, carried from frame to frame.
struct LinkShared {
    int wsum[33];
    long long wsum64[33];
    int ring_n[kRingSmem + 1], ringpre[kRingSmem + 2];
    long long counter, frame, load;
    int prevg, head, nroots, ringtot;
};

// What a run of consecutive frames works on.  A run of a whole video (or of
// the window that follows one) has spec = false and lp0 = own_g = gfirst's
// video start.  A speculative run (spec) starts `prefix` frames before the
// frames it owns with an empty state and numbers its ids from 0: its
// per-point arrays cover the points from lp0 on, the ids of the points before
// frame own_g go to its own scratch, and its state as it reaches own_g is kept
// for the comparison with the run before it.
struct LinkRun {
    uint8_t* base;      // scratch, make_lay(G, E, NP, M, spec)
    int64_t NP;         // points (and ids) the per-point arrays cover
    int64_t lp0;        // first point they cover, relative to the video
    int gfirst;         // first frame whose points can be sources
    int own_g;          // first frame whose ids the run writes to the output
    uint32_t* flags;
    long long* c0;      // spec: id counter at own_g
    bool spec;
};

// Links frames [g_lo, g_hi) of video v from the state in sh.  SEG: durations
// are left to the caller (the ids of a speculative run are not final).
template <typename SF, bool SEG>
__device__ __forceinline__ void link_frames(const LinkInput& in, const LinkLists& L, const LinkScratch& S,
                                            const LinkOutput& out, const int gb, const LinkRun& run, const int g_lo,
                                            const int g_hi, LinkShared& sh) {
    constexpr int kLinkSmemD = LinkSmem<SF>::D, kLinkSmemS = LinkSmem<SF>::S;
    const int64_t P0 = gbase(in, gb);
    const int M = in.memory, K = M + 1;
    const int G = S.max_group;
    const Lay lay = make_lay(G, S.max_edges, run.NP, M, run.spec);
    uint8_t* const base = run.base;
    int64_t* start = (int64_t*)(base + lay.start);
    int32_t* idstamp = (int32_t*)(base + lay.idstamp);
    unsigned long long* firstpos = (unsigned long long*)(base + lay.firstpos);
    // the per-point arrays, indexed by the point's place in the video
    int32_t* srcidx = (int32_t*)(base + lay.srcidx) - run.lp0;
    int32_t* srcstamp = (int32_t*)(base + lay.srcstamp) - run.lp0;
    int32_t* ring_pt = (int32_t*)(base + lay.ring_pt);
    int32_t* ring_n = (int32_t*)(base + lay.ring_n);
    int32_t* ringpre = (int32_t*)(base + lay.ringpre);
    int32_t* const g_dblk = (int32_t*)(base + lay.dblk);
    uint8_t* const g_sblk = base + lay.sblk;
    int32_t* e_src = (int32_t*)(base + lay.e_src);
    float* e_dist = (float*)(base + lay.e_dist);
    int32_t* pathD = (int32_t*)(base + lay.pathD);
    int32_t* pathS = (int32_t*)(base + lay.pathS);
    int32_t* srcLocal = (int32_t*)(base + lay.srcLocal);
    int32_t* vis_d = (int32_t*)(base + lay.vis_d);
    int32_t* vis_s = (int32_t*)(base + lay.vis_s);
    int2* stack = (int2*)(base + lay.stack);
    int32_t* r2opt = (int32_t*)(base + lay.r2a);
    int32_t* r2cho = (int32_t*)(base + lay.r2b);
    int32_t* r2best = (int32_t*)(base + lay.r2c);
    uint8_t* r2used = base + lay.r2used;
    int64_t* dur = out.dur + P0;
    int64_t* ids = out.ids;
    const int Smax = G * K;
    const float R = in.radius;
    const float R2 = __fmul_rn(R, R);
    const int tid = threadIdx.x, nth = blockDim.x;
    // shared-memory copies of the per-frame blocks (same layout as dblk / sblk)
    extern __shared__ int64_t lsm[];
    int32_t* const s_dblk = (int32_t*)lsm;                             // 10 x (kLinkSmemD + 1)
    uint8_t* const s_sblk = (uint8_t*)(s_dblk + 10 * (kLinkSmemD + 1));  // kLinkSmemS sources

    // ring sizes and their prefix live in shared memory for memory <= kRingSmem
    const bool ring_smem = M <= kRingSmem;
    int32_t* ringN = ring_smem ? sh.ring_n : ring_n;
    int32_t* ringP = ring_smem ? sh.ringpre : ringpre;
    int64_t* const pids = SEG ? (int64_t*)(base + lay.pids) - run.lp0 : nullptr;
    // first frame and point whose ids go to the output (true-state runs: all of them)
    const int32_t own_g = (SEG && run.spec) ? run.own_g : INT32_MIN;
    const int64_t own_lp = (SEG && run.spec) ? gbase(in, own_g) - P0 : INT64_MIN;
    // id of point lp of the video
    auto id_of = [&](int64_t lp) -> int64_t {
        return (SEG && lp < own_lp) ? pids[lp] : ids[P0 + lp];
    };

    for (int g = g_lo; g < g_hi; g++) {
        const int step = g - gb;
        if (!SEG && in.reset[g]) {
            // Linker::reset (src/linking.rs:401-403, src/execute_gpu.rs:792-798)
            if (tid == 0) {
                sh.counter = 0;
                sh.frame = 0;
                sh.prevg = -1;
                sh.head = 0;
            }
            for (int i = tid; i <= M; i += nth) ringN[i] = 0;
            __syncthreads();
        }
        const int64_t a = gbase(in, g);
        const int D = (int)gsize(in, g);
        const int prevg = sh.prevg;
        const int S0 = (prevg == g - 1 && prevg >= gb) ? (int)gsize(in, g - 1) : 0;
        const int64_t pa = (S0 > 0) ? gbase(in, g - 1) : 0;
        if (SEG && g == own_g) {
            int32_t* const snap_ring = (int32_t*)(base + lay.snap);
            int32_t* const snap_n = snap_ring + M * (int64_t)G;
            // the state this run reached just before its own frames
            for (int q = 0; q < M; q++) {
                const int slot = (sh.head + q) % M, n = ringN[slot];
                for (int e = tid; e < n; e += nth) snap_ring[q * G + e] = ring_pt[slot * G + e];
                if (tid == 0) snap_n[q] = n;
            }
            if (tid == 0) *run.c0 = sh.counter;
        }
        // points of frame g take their ids here, those of frame g - 1 have theirs here
        int64_t* const idg = (SEG && g < own_g) ? pids + (a - P0) : ids + a;
        const int64_t* const idp = (SEG && g - 1 < own_g) ? pids + (pa - P0) : ids + pa;
        // working arrays of this frame: shared memory when they fit
        int ring_all = 0;
        if (ring_smem)
            for (int q = 0; q < M; q++) ring_all += ringN[q];
        const bool fast = ring_smem && D <= kLinkSmemD && S0 + ring_all <= kLinkSmemS;
        const int dstr = fast ? kLinkSmemD + 1 : G + 1;
        const int sstr = fast ? kLinkSmemS : Smax;
        int32_t* const dblk = fast ? s_dblk : g_dblk;
        uint8_t* const sblk = fast ? s_sblk : g_sblk;
        SF* const sf0 = (SF*)sblk;
        SF* const sf1 = sf0 + sstr;
        int32_t* const src_pt = (int32_t*)(sf1 + sstr);
        uint8_t* const srcUsed = (uint8_t*)(src_pt + sstr);
        int32_t* const d_off = dblk;
        int32_t* const d_end = dblk + dstr;
        int32_t* const out_src = dblk + 2 * dstr;
        volatile int* const parent = (volatile int*)(dblk + 3 * dstr);
        int32_t* const comp_nd = dblk + 4 * dstr;
        int32_t* const comp_ns = dblk + 5 * dstr;
        int32_t* const comp_off = dblk + 6 * dstr;
        int32_t* const comp_soff = dblk + 7 * dstr;
        int32_t* const roots = dblk + 8 * dstr;
        int32_t* const tmp = dblk + 9 * dstr;
        // ---- P1: sources = previous frame + memory entries not already present
        for (int i0 = 2 * tid; i0 < S0; i0 += 2 * nth) {
            const int n2 = min(2, S0 - i0);
            int64_t idv[2];
#pragma unroll
            for (int u = 0; u < 2; u++)
                if (u < n2) idv[u] = idp[i0 + u];
#pragma unroll
            for (int u = 0; u < 2; u++) {
                if (u >= n2) break;
                const int i = i0 + u;
                const int64_t lp = pa + i - P0;
                idstamp[idv[u]] = step;
                src_pt[i] = (int32_t)lp;
                srcidx[lp] = i;
                srcstamp[lp] = step;
            }
        }
        if (tid == 0) {
            int tot = 0;
            for (int q = 0; q < M; q++) {
                ringP[q] = tot;
                tot += ringN[(sh.head + q) % M];
            }
            ringP[M] = tot;
            sh.ringtot = tot;
        }
        __syncthreads();
        const int RT = (M > 0) ? sh.ringtot : 0;
        // ring entries in ring order: position r -> (slot q, entry e)
        auto ring_lp = [&](int r) -> int32_t {
            int q = 0;
            while (ringP[q + 1] <= r) q++;
            const int slot = (sh.head + q) % M;
            return ring_pt[slot * G + (r - ringP[q])];
        };
        for (int r = tid; r < RT; r += nth) {
            const int64_t id = id_of(ring_lp(r));
            if (idstamp[id] != step)
                atomicMax(&firstpos[id], ((unsigned long long)(uint32_t)step << 32) | (0xFFFFFFFFull - (uint32_t)r));
        }
        __syncthreads();
        int kept_tot = 0;
        for (int base0 = 0; base0 < RT; base0 += 2 * nth) {
            int keep[2] = {0, 0};
            int32_t lpv[2] = {0, 0};
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const int r = base0 + 2 * tid + u;
                if (r < RT) {
                    lpv[u] = ring_lp(r);
                    const int64_t id = id_of(lpv[u]);
                    keep[u] = (idstamp[id] != step) &&
                              firstpos[id] ==
                                  (((unsigned long long)(uint32_t)step << 32) | (0xFFFFFFFFull - (uint32_t)r));
                }
            }
            int tot;
            const int pos = block_excl_scan(keep[0] + keep[1], &tot, sh.wsum);
#pragma unroll
            for (int u = 0; u < 2; u++) {
                if (!keep[u]) continue;
                const int si = S0 + kept_tot + pos + (u ? keep[0] : 0);
                src_pt[si] = lpv[u];
                srcidx[lpv[u]] = si;
                srcstamp[lpv[u]] = step;
            }
            kept_tot += tot;
        }
        const int Sn = S0 + kept_tot;
        __syncthreads();
        // ---- P2: destination -> source lists (ascending source index).  The
        // edges of destination j go to its own range of the frame's backward
        // lists, whose size bounds the kept edges: [d_off[j], d_end[j]).
        const int64_t fb = L.b_off[lix(L, a, K, 0)];
        if (L.b_off[lix(L, a + D, K, 0)] - fb > S.max_edges) {
            if (tid == 0) atomicOr(run.flags, in.slot_stride ? kFlagEdgeOverflow : kFlagScratch);
            return;
        }
        for (int j = tid; j < D; j += nth) {
            const int64_t pt = a + j;
            const int64_t lb = lix(L, pt, K, 0);
            int64_t bo[kLagRegs + 1];
            const bool regs = K <= kLagRegs;
#pragma unroll
            for (int i = 0; i <= kLagRegs; i++) bo[i] = (regs && i <= K) ? L.b_off[lb + i] : 0;
            const int64_t b0 = regs ? bo[0] : L.b_off[lb];
            int w = (int)(b0 - fb);
            d_off[j] = w;
            // When every lag has at most kEdgeRegs edges, all list reads are
            // issued before any write (the writes could alias them for the
            // compiler), so their latencies overlap: three dependent levels
            // instead of one chain per edge.  Same edges, same order.
            bool fits = regs;
#pragma unroll
            for (int k = 1; k <= kLagRegs; k++)
                if (k <= K && bo[k] - bo[k - 1] > kEdgeRegs) fits = false;
            if (fits) {
                int32_t ep[kLagRegs][kEdgeRegs], es[kLagRegs][kEdgeRegs];
                float ed[kLagRegs][kEdgeRegs];
#pragma unroll
                for (int k = 1; k <= kLagRegs; k++) {
                    const bool lag_on = k <= K && (k == 1 ? S0 > 0 : g - k >= run.gfirst);
#pragma unroll
                    for (int u = 0; u < kEdgeRegs; u++) {
                        const int64_t e = bo[k - 1] + u;
                        const bool on = lag_on && e < bo[k];
                        ep[k - 1][u] = on ? L.b_pts[e] : -1;
                        ed[k - 1][u] = on ? L.b_dist[e] : 0.0f;
                    }
                }
                // lags 2..K: the source's index in this step's source list,
                // or -1 when it is not a source of this step
#pragma unroll
                for (int k = 2; k <= kLagRegs; k++) {
                    const int64_t ta = (k <= K && g - k >= run.gfirst) ? gbase(in, g - k) - P0 : 0;
#pragma unroll
                    for (int u = 0; u < kEdgeRegs; u++) {
                        es[k - 1][u] = -1;
                        if (ep[k - 1][u] >= 0) {
                            const int64_t lp = ta + ep[k - 1][u];
                            const int32_t stamp = srcstamp[lp], idx = srcidx[lp];
                            es[k - 1][u] = (stamp == step) ? idx : -1;
                        }
                    }
                }
                // lag 1 (index within group g-1 == source index), then lags K..2
#pragma unroll
                for (int u = 0; u < kEdgeRegs; u++)
                    if (ep[0][u] >= 0) {
                        e_src[w] = ep[0][u];
                        e_dist[w] = ed[0][u];
                        w++;
                    }
#pragma unroll
                for (int k = kLagRegs; k >= 2; k--)
#pragma unroll
                    for (int u = 0; u < kEdgeRegs; u++)
                        if (es[k - 1][u] >= 0) {
                            e_src[w] = es[k - 1][u];
                            e_dist[w] = ed[k - 1][u];
                            w++;
                        }
                d_end[j] = w;
                parent[j] = j;
                out_src[j] = -2;
                continue;
            }
            if (S0 > 0) {
                const int64_t o1 = regs ? bo[1] : L.b_off[lb + 1];
                for (int64_t e = b0; e < o1; e++) {
                    e_src[w] = L.b_pts[e];  // index within group g-1 == source index
                    e_dist[w] = L.b_dist[e];
                    w++;
                }
            }
            // lags K..2: only sources that are in this step's source list
            auto lag = [&](int k, int64_t o0, int64_t o1) {
                const int t = g - k;
                if (t < run.gfirst) return;
                const int64_t ta = gbase(in, t) - P0;
                for (int64_t e = o0; e < o1; e++) {
                    const int64_t lp = ta + L.b_pts[e];
                    if (srcstamp[lp] == step) {
                        e_src[w] = srcidx[lp];
                        e_dist[w] = L.b_dist[e];
                        w++;
                    }
                }
            };
            if (regs) {
#pragma unroll
                for (int k = kLagRegs; k >= 2; k--)
                    if (k <= K) lag(k, bo[k - 1], bo[k]);
            } else {
                for (int k = K; k >= 2; k--) lag(k, L.b_off[lb + k - 1], L.b_off[lb + k]);
            }
            d_end[j] = w;
            parent[j] = j;
            out_src[j] = -2;
        }
        // ---- P3: trivial links and subnets (connected components)
        // forward range of every source toward this frame, read once
        for (int s = tid; s < Sn; s += nth) {
            const int64_t pt = P0 + src_pt[s];
            const int64_t l = lix(L, pt, K, g - ggroup(in, pt) - 1);
            const int64_t f0 = L.f_off[l], f1 = L.f_off[l + 1];
            sf0[s] = (SF)f0;
            sf1[s] = (SF)f1;
            srcUsed[s] = 0;
        }
        __syncthreads();
        for (int s = tid; s < Sn; s += nth) {
            const int64_t f0 = sf0[s], f1 = sf1[s];
            if (f1 - f0 >= 2) {
                const int j0 = L.f_pts[f0];
                for (int64_t e = f0 + 1; e < f1; e++) uf_union(parent, j0, L.f_pts[e]);
            }
        }
        for (int j = tid; j < D; j += nth) {
            const int e0 = d_off[j], deg = d_end[j] - e0;
            if (deg == 0) {
                out_src[j] = -1;
            } else if (deg == 1) {
                const int s = e_src[e0];
                if (sf1[s] - sf0[s] == 1) out_src[j] = s;
            }
        }
        __syncthreads();
        for (int j = tid; j < D; j += nth) {
            tmp[j] = uf_find(parent, j);
            comp_nd[j] = 0;
            comp_ns[j] = 0;
        }
        __syncthreads();
        for (int j = tid; j < D; j += nth)
            if (out_src[j] == -2) atomicAdd(&comp_nd[tmp[j]], 1);
        for (int s = tid; s < Sn; s += nth) {
            const int64_t f0 = sf0[s];
            if (sf1[s] > f0) {
                const int j0 = L.f_pts[f0];
                if (out_src[j0] == -2) atomicAdd(&comp_ns[tmp[j0]], 1);
            }
        }
        __syncthreads();
        {
            // one 64-bit scan of (roots, destinations) and one of sources, two
            // destinations per thread in destination order
            long long acc_rd = 0;
            int offs = 0;
            for (int base0 = 0; base0 < D; base0 += 2 * nth) {
                int isroot[2], nd[2], ns[2];
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    const int j = base0 + 2 * tid + u;
                    isroot[u] = (j < D && out_src[j] == -2 && tmp[j] == j) ? 1 : 0;
                    nd[u] = isroot[u] ? comp_nd[j] : 0;
                    ns[u] = isroot[u] ? comp_ns[j] : 0;
                }
                const long long rd0 = (long long)isroot[0] + ((long long)nd[0] << 32);
                const long long rd1 = (long long)isroot[1] + ((long long)nd[1] << 32);
                long long trd;
                int ts;
                const long long prd = block_excl_scan64(rd0 + rd1, &trd, sh.wsum64);
                const int ps = block_excl_scan(ns[0] + ns[1], &ts, sh.wsum);
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    if (!isroot[u]) continue;
                    const int j = base0 + 2 * tid + u;
                    const long long pr_ = acc_rd + prd + (u ? rd0 : 0);
                    roots[(int)(pr_ & 0xFFFFFFFFll)] = j;
                    comp_off[j] = (int)(pr_ >> 32);
                    comp_soff[j] = offs + ps + (u ? ns[0] : 0);
                }
                acc_rd += trd;
                offs += ts;
            }
            if (tid == 0) {
                sh.nroots = (int)(acc_rd & 0xFFFFFFFFll);
                sh.load = 0;
            }
        }
        __syncthreads();
        const int nroots = sh.nroots;
        // ---- P4: the reference's DFS order per subnet (recurse, linking.rs:595-621)
        for (int q = tid; q < nroots; q += nth) {
            const int r = roots[q];
            const int od = comp_off[r], os = comp_soff[r];
            int2* stk = stack + od + os;
            int nd = 0, ns = 0, sp = 0;
            vis_d[r] = step;
            pathD[od + nd++] = r;
            stk[sp++] = make_int2(r, 0);  // (node, next edge); dests tagged by >= 0 side bit below
            // side encoding: dest nodes stored as node, sources as -(node+1)
            while (sp > 0) {
                int2& top = stk[sp - 1];
                if (top.x >= 0) {  // destination: its sources in list order
                    const int j = top.x;
                    const int e0 = d_off[j], e1 = d_end[j];
                    bool pushed = false;
                    while (e0 + top.y < e1) {
                        int s = e_src[e0 + top.y];
                        top.y++;
                        if (vis_s[s] != step) {
                            vis_s[s] = step;
                            srcLocal[s] = ns;
                            pathS[os + ns++] = s;
                            stk[sp++] = make_int2(-(s + 1), 0);
                            pushed = true;
                            break;
                        }
                    }
                    if (!pushed) sp--;
                } else {  // source: its destinations in list order
                    const int s = -top.x - 1;
                    const int64_t f0 = sf0[s], f1 = sf1[s];
                    bool pushed = false;
                    while (f0 + top.y < f1) {
                        int j = L.f_pts[f0 + top.y];
                        top.y++;
                        if (vis_d[j] != step) {
                            vis_d[j] = step;
                            pathD[od + nd++] = j;
                            stk[sp++] = make_int2(j, 0);
                            pushed = true;
                            break;
                        }
                    }
                    if (!pushed) sp--;
                }
            }
            if (nd > 1) atomicAdd((unsigned long long*)&sh.load, (unsigned long long)((long long)nd * ns));
        }
        __syncthreads();
        if (sh.load > 5000) {
            // TooDenseToLink (src/linking.rs:677-682)
            if (tid == 0) atomicOr(run.flags, kFlagTooDense);
            return;
        }
        // ---- P5: branch and bound per subnet (recurse2, linking.rs:687-766)
        bool spent = false;   // a subnet of this thread's ran out of steps
        for (int q = tid; q < nroots; q += nth) {
            const int r = roots[q];
            const int od = comp_off[r], os = comp_soff[r];
            const int nd = comp_nd[r], ns = comp_ns[r];
            int* opt = r2opt + od;
            int* cho = r2cho + od;
            int* bst = r2best + od;
            uint8_t* used = r2used + os;
            for (int i = 0; i < ns; i++) used[i] = 0;
            float score = 0.0f, best = INFINITY;
            bool has_best = false;
            long long budget = 0;
            int level = 0;
            opt[0] = 0;
            bool over = false;
            while (true) {
                if (++budget > kSubnetBudget) { over = true; break; }
                const int j = pathD[od + level];
                const int e0 = d_off[j];
                const int deg = d_end[j] - e0;
                const int o = opt[level];
                bool ascend = false;
                if (o > deg) {
                    ascend = true;
                } else if (score > best) {
                    ascend = true;
                } else {
                    const bool is_null = (o == deg);
                    const float c = is_null ? R2 : e_dist[e0 + o];
                    score = __fadd_rn(score, c);
                    int ls = -1;
                    if (!is_null) {
                        ls = srcLocal[e_src[e0 + o]];
                        if (used[ls]) {
                            score = __fsub_rn(score, c);
                            opt[level] = o + 1;
                            continue;
                        }
                        used[ls] = 1;
                    }
                    cho[level] = ls;
                    if (level == nd - 1) {
                        if (score < best) {
                            best = score;
                            has_best = true;
                            for (int l = 0; l < nd; l++) bst[l] = cho[l];
                        }
                        if (!is_null) used[ls] = 0;
                        score = __fsub_rn(score, c);
                        opt[level] = o + 1;
                    } else {
                        level++;
                        opt[level] = 0;
                    }
                    continue;
                }
                if (ascend) {
                    level--;
                    if (level < 0) break;
                    const int jp = pathD[od + level];
                    const int ep = d_off[jp];
                    const int degp = d_end[jp] - ep;
                    const int op = opt[level];
                    const bool nullp = (op == degp);
                    const float cp = nullp ? R2 : e_dist[ep + op];
                    if (!nullp) used[cho[level]] = 0;
                    score = __fsub_rn(score, cp);
                    opt[level] = op + 1;
                }
            }
            spent |= over;
            for (int l = 0; l < nd; l++) {
                int ch = has_best ? bst[l] : -1;
                out_src[pathD[od + l]] = (ch >= 0) ? pathS[os + ch] : -1;
            }
        }
        if (__syncthreads_or(spent)) {
            if (tid == 0) atomicOr(run.flags, kFlagSubnetBudget);
            return;
        }
        // ---- P6: ids (new ones in destination order, src/linking.rs:788-798)
        {
            int newtot = 0;
            const long long counter = sh.counter;
            const long long frame = sh.frame;
            for (int base0 = 0; base0 < D; base0 += 2 * nth) {
                int osrc[2], isnew[2];
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    const int j = base0 + 2 * tid + u;
                    osrc[u] = (j < D) ? out_src[j] : 0;
                    isnew[u] = (j < D && osrc[u] < 0) ? 1 : 0;
                }
                int tot;
                const int pos = block_excl_scan(isnew[0] + isnew[1], &tot, sh.wsum);
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    const int j = base0 + 2 * tid + u;
                    if (j >= D) break;
                    if (isnew[u]) {
                        const long long id = counter + newtot + pos + (u ? isnew[0] : 0);
                        idg[j] = id;
                        if (!SEG) start[id] = frame;
                    } else {
                        const int s = osrc[u];
                        idg[j] = id_of(src_pt[s]);
                        srcUsed[s] = 1;
                    }
                }
                newtot += tot;
            }
            __syncthreads();
            if (tid == 0) sh.counter = counter + newtot;
        }
        // ---- P7: memory ring and durations (src/linking.rs:481-503)
        {
            const long long frame = sh.frame;
            if (M > 0) {
                const int hs = sh.head;
                const int nleave = ringN[hs];
                for (int e = tid; !SEG && e < nleave; e += nth) {
                    int64_t id = ids[P0 + ring_pt[hs * G + e]];
                    dur[id] = (frame - start[id]) - M;
                }
                __syncthreads();
                int ut = 0;
                for (int base0 = 0; base0 < S0; base0 += 2 * nth) {
                    int un[2];
#pragma unroll
                    for (int u = 0; u < 2; u++) {
                        const int s = base0 + 2 * tid + u;
                        un[u] = (s < S0 && !srcUsed[s]) ? 1 : 0;
                    }
                    int tot;
                    const int pos = block_excl_scan(un[0] + un[1], &tot, sh.wsum);
#pragma unroll
                    for (int u = 0; u < 2; u++)
                        if (un[u]) ring_pt[hs * G + ut + pos + (u ? un[0] : 0)] = src_pt[base0 + 2 * tid + u];
                    ut += tot;
                }
                if (tid == 0) {
                    ringN[hs] = ut;
                    sh.head = (hs + 1) % M;
                }
            } else if (!SEG) {
                for (int s = tid; s < S0; s += nth) {
                    if (!srcUsed[s]) {
                        int64_t id = ids[P0 + src_pt[s]];
                        dur[id] = frame - start[id];
                    }
                }
            }
            __syncthreads();
            if (tid == 0) {
                sh.prevg = g;
                sh.frame = frame + 1;
            }
            __syncthreads();
        }
    }
}

// Whether the video's linking has stopped, the same answer for every thread of
// the block: the CTA of the video's first segment and the list kernels of the
// next window raise flags while this one runs, so a thread's own read must not
// decide about a barrier.  Whole block; `sh` is free again at the next barrier
// after the call.
__device__ __forceinline__ bool link_stopped(const uint32_t* flags, int* sh) {
    __syncthreads();
    if (threadIdx.x == 0) *sh = (*(const volatile uint32_t*)flags & kLinkStopFlags) != 0 ? 1 : 0;
    __syncthreads();
    return *sh != 0;
}

// Every video (or the next window of one) by one CTA, frame after frame.
template <typename SF>
__global__ void __launch_bounds__(kLinkThreads)
link_video_kernel(LinkInput in, LinkLists L, LinkScratch S, LinkOutput out, LinkWindow W) {
    __shared__ LinkShared sh;
    __shared__ int sh_stop;
    const int v = blockIdx.x;
    const int gb = in.vgrp[v], ge = in.vgrp[v + 1];
    const int g_lo = (W.g0 < 0) ? gb : W.g0, g_hi = (W.g0 < 0) ? ge : W.g1;
    if (link_stopped(out.flags + v, &sh_stop)) return;  // an earlier window stopped this video
    const int64_t P0 = gbase(in, gb);
    const int64_t NP = in.slot_stride ? (int64_t)(ge - gb) * in.slot_stride : in.goff[ge] - P0;
    const int M = in.memory, K = M + 1;
    const int G = S.max_group;
    const Lay lay = make_lay(G, S.max_edges, S.max_points, M, false);
    uint8_t* base = S.base + (size_t)v * S.bytes_per_video;
    const int64_t* start = (const int64_t*)(base + lay.start);
    int32_t* idstamp = (int32_t*)(base + lay.idstamp);
    unsigned long long* firstpos = (unsigned long long*)(base + lay.firstpos);
    int32_t* srcstamp = (int32_t*)(base + lay.srcstamp);
    int32_t* ring_pt = (int32_t*)(base + lay.ring_pt);
    int32_t* ring_n = (int32_t*)(base + lay.ring_n);
    int32_t* vis_d = (int32_t*)(base + lay.vis_d);
    int32_t* vis_s = (int32_t*)(base + lay.vis_s);
    int64_t* dur = out.dur + P0;
    int64_t* ids = out.ids;
    const int Smax = G * K;
    const int tid = threadIdx.x, nth = blockDim.x;
    const bool ring_smem = M <= kRingSmem;
    int32_t* ringN = ring_smem ? sh.ring_n : ring_n;
    if (W.first) {
        if (W.init_points) {
            for (int64_t i = tid; i < NP; i += nth) {
                idstamp[i] = -1;
                srcstamp[i] = -1;
                firstpos[i] = 0ull;
            }
        }
        for (int i = tid; i < Smax; i += nth) vis_s[i] = -1;
        for (int i = tid; i < G; i += nth) vis_d[i] = -1;
        for (int i = tid; i <= M; i += nth) ringN[i] = 0;
        if (tid == 0) {
            sh.counter = 0;
            sh.frame = 0;
            sh.prevg = -1;
            sh.head = 0;
        }
    } else {
        if (ring_smem)
            for (int i = tid; i <= M; i += nth) ringN[i] = ring_n[i];
    }
    if (!W.first && tid == 0) {
        const LinkState st = W.state[v];
        sh.counter = st.counter;
        sh.frame = st.frame;
        sh.prevg = st.prevg;
        sh.head = st.head;
    }
    __syncthreads();

    LinkRun run;
    run.base = base;
    run.NP = S.max_points;
    run.lp0 = 0;
    run.gfirst = gb;
    run.own_g = gb;
    run.flags = out.flags + v;
    run.c0 = nullptr;
    run.spec = false;
    link_frames<SF, false>(in, L, S, out, gb, run, g_lo, g_hi, sh);
    const bool stopped = link_stopped(out.flags + v, &sh_stop);
    if (!W.last) {
        if (ring_smem)
            for (int i = tid; i <= M; i += nth) ring_n[i] = ringN[i];
        if (tid == 0 && !stopped) {
            LinkState st;
            st.counter = sh.counter;
            st.frame = sh.frame;
            st.prevg = sh.prevg;
            st.head = sh.head;
            W.state[v] = st;
        }
        return;
    }
    // ---- Linker::finish (src/linking.rs:505-520)
    if (!stopped) {
        const long long frame = sh.frame;
        if (M > 0) {
            for (int q = 0; q < M; q++) {
                int slot = (sh.head + q) % M;
                int n = ringN[slot];
                for (int e = tid; e < n; e += nth) {
                    int64_t id = ids[P0 + ring_pt[slot * G + e]];
                    dur[id] = (frame - start[id]) - (M - q);
                }
                __syncthreads();
            }
        }
        if (sh.prevg >= gb) {
            const int pg = sh.prevg;
            const int64_t pb = gbase(in, pg), pe = pb + gsize(in, pg);
            for (int64_t p = pb + tid; p < pe; p += nth) {
                int64_t id = ids[p];
                dur[id] = frame - start[id];
            }
        }
    }
    if (tid == 0) out.counter[v] = sh.counter;
}

// ------------------------------------------------------ segments of a video
// The frame loop is serial (30-57 us a frame in one CTA), but what a frame
// takes from the frames before it is only the detections of the last one and
// the memory ring, and the linker compares ids for nothing but identity.  So
// the frames are cut into segments of Q.len frames, one CTA each.  The first
// runs from the true state; each other one starts Q.prefix frames early from
// an empty state, which the prefix replaces by the true one up to the names
// of the ids: old entries are out of the ring after memory + 1 frames, and a
// match they would have changed stops mattering soon after.  Of the two runs
// at a boundary the one that ends later compares them: where the state the
// later segment had reached holds the same detections in the same ring order
// as the end of the one before, with ids that correspond one to one, every
// later match is the sequential linker's, and the segment's ids are its own
// ones renamed: those of the boundary's detections by that correspondence, the
// new ones by an offset.  The CTA that ends last adds the offsets up, and links
// a segment whose boundary does not hold again from the true state.  The
// result is the sequential linker's in every case, a boundary that does not
// hold costs its frames.
// Measured on a B200, one video: 400 frames of 2000 given points, memory 3,
// 16.4 ms in one CTA and 0.98 ms here (80 segments of 5 frames, each run with a
// prefix of 10; 1.55 ms where the points mix freely); 512 located frames of
// 2048^2 with 2000 spots: 4.4 ms of linking left after the last frame is located
// and 1 ms here.  Boundaries that did not hold, freely mixing points, step 1.4
// px: none of 79 at search_range 7 or 9, 7 of 79 at search_range 5 (4.3 ms); none
// with memory 0 or 1.

// Points of frames [g0, g1).
__device__ __forceinline__ int64_t frames_points(const LinkInput& in, int g0, int g1) {
    if (!in.slot_stride) return in.goff[g1] - in.goff[g0];
    int64_t n = 0;
    for (int g = g0; g < g1; g++) n += in.gcount[g];
    return n;
}

// Where the runs of a video keep what joins them.  A speculative run's
// first ids (those of the boundary it starts at) have partners in the run
// before: partner[id] in the lower half of its unused start array; the upper
// half takes, for the comparison at its end, the later run's id of each of its
// own.
struct SegmentRuns {
    LinkSeg* seg;
    uint8_t *mbase, *qbase;      // true-state scratch, speculative runs' scratch of the video
    size_t bytes;
    int64_t mNP, qNP;
    size_t m_start, q_start;
    __device__ __forceinline__ uint8_t* spec(int t) const { return qbase + (size_t)(t - 1) * bytes; }
    __device__ __forceinline__ int32_t* partner(int t) const { return (int32_t*)(spec(t) + q_start); }
    // the comparison array of the run that ended segment t
    __device__ __forceinline__ int32_t* inverse(int t, bool true_run) const {
        return true_run ? (int32_t*)(mbase + m_start) + mNP : (int32_t*)(spec(t) + q_start) + qNP;
    }
    // final id of an id of segment t: back through the boundaries to the
    // segment that gave it
    __device__ __forceinline__ int64_t final_id(int t, int64_t id) const {
        while (!__ldcg(&seg[t].final_ids)) {
            const long long c0 = __ldcg(&seg[t].c0);
            if (id >= c0) return __ldcg(&seg[t].base) + (id - c0);
            id = __ldcg(partner(t) + id);
            t--;
        }
        return id;
    }
};

// 640 threads: most of a frame is latency and barriers, and the frame loop
// spills at the 64 registers of 1024.  Device time of the segments (B200) with
// 512 / 640 / 768 / 1024 threads: 400 frames of 2000 points, memory 3, 1230 /
// 1173 / 1177 / 1178 us; 160 frames of 500, memory 2, beside locating 689 /
// 676 / 737 / 870; 64 frames of 4000, memory 3, 1633 / 1479 / 1405 / 1335.
constexpr int kSegThreads = 640;
template <typename SF>
__global__ void __launch_bounds__(kSegThreads)
link_segments_kernel(LinkInput in, LinkLists L, LinkScratch S, LinkOutput out, LinkWindow W, LinkSegs Q) {
    __shared__ LinkShared sh;
    __shared__ int sh_last;
    const int v = blockIdx.y, s = blockIdx.x;
    const int gb = in.vgrp[v], ge = in.vgrp[v + 1];
    const int w_lo = (W.g0 < 0) ? gb : W.g0, w_hi = (W.g0 < 0) ? ge : W.g1;
    const int nseg = max(1, (w_hi - w_lo + Q.len - 1) / Q.len);
    if (s >= nseg) return;
    const int64_t P0 = gbase(in, gb);
    const int M = in.memory, K = M + 1;
    const int G = S.max_group, Smax = G * K;
    const int tid = threadIdx.x, nth = blockDim.x;
    LinkSeg* const seg = Q.seg + (size_t)v * Q.max_segs;
    int64_t* const ids = out.ids;
    auto seg_first = [&](int t) { return w_lo + t * Q.len; };
    auto seg_end = [&](int t) { return min(w_lo + (t + 1) * Q.len, w_hi); };
    // the true-state scratch, and that of the speculative run of segment t >= 1
    uint8_t* const mbase = S.base + (size_t)v * S.bytes_per_video;
    const Lay ml = make_lay(G, S.max_edges, S.max_points, M, false);
    const Lay pl = make_lay(G, S.max_edges, Q.points, M, true);
    SegmentRuns runs;
    runs.seg = seg;
    runs.mbase = mbase;
    runs.qbase = Q.base + (size_t)v * (Q.max_segs - 1) * Q.bytes;
    runs.bytes = Q.bytes;
    runs.mNP = S.max_points;
    runs.qNP = Q.points;
    runs.m_start = ml.start;
    runs.q_start = pl.start;
    auto spec_base = [&](int t) { return runs.spec(t); };
    int32_t* const m_ring = (int32_t*)(mbase + ml.ring_pt);
    int32_t* const m_ring_n = (int32_t*)(mbase + ml.ring_n);

    __shared__ LinkRun run;   // in shared memory: the frame loop needs every register
    __shared__ int sh_lo, sh_hi;
    // clears the stamps that a run from the true state (in sh and the ring)
    // over segment t reads before it writes them
    auto begin_true = [&](int t) {
        const int g_lo = seg_first(t), g_hi = seg_end(t);
        if (tid == 0) {
            sh_lo = g_lo;
            sh_hi = g_hi;
            run.base = mbase;
            run.NP = S.max_points;
            run.lp0 = 0;
            run.gfirst = gb;
            run.own_g = gb;
            run.flags = out.flags + v;
            run.c0 = nullptr;
            run.spec = false;
        }
        int32_t* const idstamp = (int32_t*)(mbase + ml.idstamp);
        int32_t* const srcstamp = (int32_t*)(mbase + ml.srcstamp);
        unsigned long long* const firstpos = (unsigned long long*)(mbase + ml.firstpos);
        if (g_hi > g_lo) {
            const int64_t q0 = gbase(in, max(gb, g_lo - K)) - P0;
            const int64_t q1 = gbase(in, g_hi - 1) + gsize(in, g_hi - 1) - P0;
            for (int64_t i = q0 + tid; i < q1; i += nth) srcstamp[i] = -1;
            const int64_t c = sh.counter, n = frames_points(in, g_lo, g_hi);
            for (int64_t i = tid; i < n; i += nth) {
                idstamp[c + i] = -1;
                firstpos[c + i] = 0ull;
            }
            if (sh.prevg == g_lo - 1 && sh.prevg >= gb) {
                const int64_t pa = gbase(in, sh.prevg), pn = gsize(in, sh.prevg);
                for (int64_t i = tid; i < pn; i += nth) {
                    const int64_t id = __ldcg(ids + pa + i);
                    idstamp[id] = -1;
                    firstpos[id] = 0ull;
                }
            }
            for (int q = 0; q < M; q++)
                for (int e = tid; e < sh.ring_n[q]; e += nth) {
                    const int64_t id = __ldcg(ids + P0 + m_ring[q * G + e]);
                    idstamp[id] = -1;
                    firstpos[id] = 0ull;
                }
        }
    };
    // A window that stopped has left no state for the next one.  (The counts of
    // arrivals that this leaves open are cleared before the next call's first
    // launch; until then every CTA returns here.)
    if (link_stopped(out.flags + v, &sh_last)) return;
    if (tid == 0) {
        seg[s].flags = 0;
        seg[s].c0 = 0;
        sh.counter = 0;
        sh.frame = 0;
        sh.prevg = -1;
        sh.head = 0;
        if (s == 0 && !W.first) {
            const LinkState st = W.state[v];
            sh.counter = st.counter;
            sh.prevg = st.prevg;
            sh.head = st.head;
        }
    }
    for (int i = tid; i <= M; i += nth) sh.ring_n[i] = (s == 0 && !W.first) ? m_ring_n[i] : 0;
    if (s == 0 && W.first) {
        int32_t* const vis_d = (int32_t*)(mbase + ml.vis_d);
        int32_t* const vis_s = (int32_t*)(mbase + ml.vis_s);
        for (int i = tid; i < Smax; i += nth) vis_s[i] = -1;
        for (int i = tid; i < G; i += nth) vis_d[i] = -1;
    }
    __syncthreads();
    if (s == 0) {
        begin_true(0);
    } else {
        const int g_lo = max(seg_first(s) - Q.prefix, w_lo), g_hi = seg_end(s);
        uint8_t* const b = spec_base(s);
        if (tid == 0) {
            sh_lo = g_lo;
            sh_hi = g_hi;
            run.base = b;
            run.NP = Q.points;
            run.lp0 = gbase(in, g_lo) - P0;
            run.gfirst = g_lo;
            run.own_g = seg_first(s);
            run.flags = &seg[s].flags;
            run.c0 = &seg[s].c0;
            run.spec = true;
        }
        int32_t* const idstamp = (int32_t*)(b + pl.idstamp);
        int32_t* const srcstamp = (int32_t*)(b + pl.srcstamp);
        unsigned long long* const firstpos = (unsigned long long*)(b + pl.firstpos);
        int32_t* const vis_d = (int32_t*)(b + pl.vis_d);
        int32_t* const vis_s = (int32_t*)(b + pl.vis_s);
        const int64_t nlp = gbase(in, g_hi - 1) + gsize(in, g_hi - 1) - gbase(in, g_lo);
        for (int64_t i = tid; i < nlp; i += nth) srcstamp[i] = -1;
        const int64_t n = frames_points(in, g_lo, g_hi);
        for (int64_t i = tid; i < n; i += nth) {
            idstamp[i] = -1;
            firstpos[i] = 0ull;
        }
        for (int i = tid; i < Smax; i += nth) vis_s[i] = -1;
        for (int i = tid; i < G; i += nth) vis_d[i] = -1;
    }
    __syncthreads();

    link_frames<SF, true>(in, L, S, out, gb, run, sh_lo, sh_hi, sh);
    __syncthreads();
    {
        int32_t* const rn = (int32_t*)(run.base + (run.spec ? pl.ring_n : ml.ring_n));
        for (int i = tid; i <= M; i += nth) rn[i] = sh.ring_n[i];
        if (tid == 0) {
            seg[s].counter = sh.counter;
            seg[s].head = sh.head;
            seg[s].final_ids = run.spec ? 0 : 1;
            seg[s].base = 0;
        }
    }
    // Compares the end of segment t - 1 (its run in the true-state scratch, or
    // the speculative one) with the state that segment t's run had reached:
    // the same detections in ring order, ids one to one.  Leaves the partners.
    // Whole block.
    __shared__ int sh_pre[kRingSmem + 2];
    auto joins = [&](int t, bool true_run) -> bool {
        uint8_t* const cb = true_run ? mbase : runs.spec(t - 1);
        const uint8_t* const tb = runs.spec(t);
        const int32_t* const c_ring = (const int32_t*)(cb + (true_run ? ml.ring_pt : pl.ring_pt));
        const int32_t* const c_ring_n = (const int32_t*)(cb + (true_run ? ml.ring_n : pl.ring_n));
        const int32_t* const t_ring = (const int32_t*)(tb + pl.snap);
        const int32_t* const t_ring_n = t_ring + M * (int64_t)G;
        const int64_t* const t_pids = (const int64_t*)(tb + pl.pids);
        int32_t* const partner = runs.partner(t);
        int32_t* const inverse = runs.inverse(t - 1, true_run);
        const int ta = seg_first(t), head = __ldcg(&seg[t - 1].head);
        const int64_t t_lp0 = gbase(in, max(ta - Q.prefix, w_lo)) - P0;
        const int64_t pa = gbase(in, ta - 1) - P0;
        const int pn = (int)gsize(in, ta - 1);
        __syncthreads();
        if (tid == 0) {
            // detections of the last frame, then the ring's by age
            // (a run that raised a flag has no state)
            bool same = __ldcg(&seg[t].flags) == 0 && (true_run || __ldcg(&seg[t - 1].flags) == 0) &&
                        !(__ldcg(out.flags + v) & kLinkStopFlags);
            int tot = pn;
            for (int q = 0; q < M; q++) {
                sh_pre[q] = tot;
                const int n = __ldcg(t_ring_n + q);
                if (__ldcg(c_ring_n + (head + q) % M) != n) same = false;
                tot += n;
            }
            sh_pre[M] = same ? tot : -1;
        }
        __syncthreads();
        const int tot = sh_pre[M];
        if (tot < 0) return false;
        for (int pass = 0; pass < 2; pass++) {
            bool ok = true;
            for (int e = tid; e < tot; e += nth) {
                int64_t lp = pa + e;
                if (e >= pn) {
                    int q = 0;
                    while (sh_pre[q + 1] <= e) q++;
                    const int32_t a = __ldcg(c_ring + ((head + q) % M) * (int64_t)G + (e - sh_pre[q]));
                    if (a != __ldcg(t_ring + q * (int64_t)G + (e - sh_pre[q]))) {
                        ok = false;
                        break;
                    }
                    lp = a;
                }
                const int32_t idc = (int32_t)__ldcg(ids + P0 + lp), idt = (int32_t)__ldcg(t_pids + lp - t_lp0);
                if (pass == 0) {
                    partner[idt] = idc;
                    inverse[idc] = idt;
                } else {
                    ok &= __ldcg(partner + idt) == idc && __ldcg(inverse + idc) == idt;
                }
            }
            __threadfence_block();
            if (!__syncthreads_and(ok)) return false;
        }
        return true;
    };
    // the later of the two runs at a boundary compares them
    for (int t = max(s, 1); t <= min(s + 1, nseg - 1); t++) {
        __syncthreads();
        if (tid == 0) {
            __threadfence();
            sh_last = atomicAdd(&seg[t].met, 1) == 1 ? 1 : 0;
            __threadfence();
        }
        __syncthreads();
        if (!sh_last) continue;
        const bool ok = joins(t, t == 1);
        if (tid == 0) {
            seg[t].joined = ok ? 1 : 0;
            seg[t].met = 0;
        }
    }
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        sh_last = atomicAdd(Q.arrived + v, 1u) == (uint32_t)nseg - 1u ? 1 : 0;
        __threadfence();
    }
    __syncthreads();
    if (!sh_last) return;

    // ---- the last CTA joins the segments in order
    if (tid == 0) Q.arrived[v] = 0;
    if (link_stopped(out.flags + v, &sh_last)) return;
    int cur = 0;               // last segment whose ids are known
    bool cur_true = true;      // its run worked in the true-state scratch
    bool again = false;        // it was linked a second time
    long long gcount = __ldcg(&seg[0].counter);   // ids given so far
    for (int t = 1; t < nseg; t++) {
        if (again ? joins(t, true) : __ldcg(&seg[t].joined) != 0) {
            if (tid == 0) seg[t].base = gcount;
            gcount += __ldcg(&seg[t].counter) - __ldcg(&seg[t].c0);
            cur = t;
            cur_true = false;
            again = false;
            continue;
        }
        // final ids for all of segment cur, its ring to the true-state
        // scratch, and segment t once more from there
        uint8_t* const cb = cur_true ? mbase : runs.spec(cur);
        const int32_t* const c_ring = (const int32_t*)(cb + (cur_true ? ml.ring_pt : pl.ring_pt));
        const int32_t* const c_ring_n = (const int32_t*)(cb + (cur_true ? ml.ring_n : pl.ring_n));
        const int head = __ldcg(&seg[cur].head);
        __syncthreads();
        if (!cur_true) {
            for (int g = seg_first(cur); g < seg_first(t); g++) {
                const int64_t x = gbase(in, g), n = gsize(in, g);
                for (int64_t i = x + tid; i < x + n; i += nth) ids[i] = runs.final_id(cur, __ldcg(ids + i));
            }
            for (int q = 0; q < M; q++) {
                const int n = __ldcg(c_ring_n + q);
                for (int e = tid; e < n; e += nth) m_ring[q * G + e] = __ldcg(c_ring + q * (int64_t)G + e);
            }
        }
        for (int i = tid; i <= M; i += nth) sh.ring_n[i] = __ldcg(c_ring_n + i);
        __syncthreads();
        if (tid == 0) {
            seg[cur].final_ids = 1;
            sh.counter = gcount;
            sh.prevg = seg_first(t) - 1;
            sh.head = head;
        }
        __syncthreads();
        begin_true(t);
        __syncthreads();
        link_frames<SF, true>(in, L, S, out, gb, run, sh_lo, sh_hi, sh);
        if (link_stopped(out.flags + v, &sh_last)) return;
        gcount = sh.counter;
        for (int i = tid; i <= M; i += nth) m_ring_n[i] = sh.ring_n[i];
        if (tid == 0) {
            seg[t].head = sh.head;
            seg[t].counter = gcount;
            seg[t].final_ids = 1;
            if (Q.again) atomicAdd(Q.again + (W.last ? 1 : 0), 1u);
        }
        cur = t;
        cur_true = true;
        again = true;
        __syncthreads();
    }
    // the state the next window starts from
    if (!W.last && !cur_true) {
        const uint8_t* const cb = spec_base(cur);
        const int32_t* const c_ring = (const int32_t*)(cb + pl.ring_pt);
        const int32_t* const c_ring_n = (const int32_t*)(cb + pl.ring_n);
        for (int q = 0; q < M; q++) {
            const int n = __ldcg(c_ring_n + q);
            for (int e = tid; e < n; e += nth) m_ring[q * G + e] = __ldcg(c_ring + q * (int64_t)G + e);
        }
        for (int i = tid; i <= M; i += nth) m_ring_n[i] = __ldcg(c_ring_n + i);
    }
    if (tid == 0) {
        if (W.last) {
            out.counter[v] = gcount;
        } else {
            LinkState st;
            st.counter = gcount;
            st.frame = 0;
            st.prevg = w_hi - 1;
            st.head = __ldcg(&seg[cur].head);
            W.state[v] = st;
        }
    }
}

// Final ids of the points of a window whose segments are resolved and, with
// out.dur_range, the frames their ids were first and last seen in.
__global__ void segment_ids_kernel(LinkInput in, LinkScratch S, LinkOutput out, LinkWindow W, LinkSegs Q, int64_t p0,
                                   int64_t p1) {
    const int64_t p = p0 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= p1) return;
    const int g = ggroup(in, p);
    if (in.slot_stride && p - gbase(in, g) >= gsize(in, g)) return;  // empty slot
    int x = 0, y = in.nvideos;
    while (y - x > 1) {
        const int m = (x + y) >> 1;
        if (in.vgrp[m] <= g) x = m; else y = m;
    }
    const int v = x;
    if (out.flags[v] & kLinkStopFlags) return;
    const int gb = in.vgrp[v];
    const int w_lo = (W.g0 < 0) ? gb : W.g0;
    const int t = (g - w_lo) / Q.len;
    const LinkSeg q = Q.seg[(size_t)v * Q.max_segs + t];
    int64_t id = out.ids[p];
    if (!q.final_ids) {
        const Lay pl = make_lay(S.max_group, S.max_edges, Q.points, in.memory, true);
        SegmentRuns runs;
        runs.seg = Q.seg + (size_t)v * Q.max_segs;
        runs.qbase = Q.base + (size_t)v * (Q.max_segs - 1) * Q.bytes;
        runs.bytes = Q.bytes;
        runs.q_start = pl.start;
        id = runs.final_id(t, id);
        out.ids[p] = id;
    }
    if (out.dur_range) {
        int32_t* const r = (int32_t*)(out.dur + gbase(in, gb) + id);
        atomicMax(r, INT32_MAX - (g - gb));
        atomicMax(r + 1, g - gb + 1);
    }
}

// Duration of an id from its entry: as the sequential linker writes it, or
// from the first and last frame.
__device__ __forceinline__ int64_t id_duration(const LinkOutput& out, int64_t at) {
    if (!out.dur_range) return out.dur[at];
    const int32_t* const r = (const int32_t*)(out.dur + at);
    return (int64_t)r[1] - (int64_t)(INT32_MAX - r[0]);
}

// Per-row durations through the reference's f32 round trip of the particle
// id (src/execute_gpu.rs:812-815, 1165-1181).
__global__ void durations_kernel(LinkInput in, LinkOutput out, int64_t* row_dur) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= in.npoints) return;
    const int h = in.pgroup[p];
    int x = 0, y = in.nvideos;
    while (y - x > 1) {
        int m = (x + y) >> 1;
        if (in.vgrp[m] <= h) x = m; else y = m;
    }
    const int v = x;
    const int64_t P0 = in.goff[in.vgrp[v]];
    const int64_t id = (int64_t)(float)out.ids[p];
    if ((uint64_t)id >= (uint64_t)out.counter[v]) {
        atomicOr(out.flags + v, kFlagScratch);
        row_dur[p] = -1;
        return;
    }
    row_dur[p] = id_duration(out, P0 + id);
}

// Slot mode: the table rows of every point (row_off[g] + j) receive the
// particle id after the reference's f32 round trip and its duration
// (src/execute_gpu.rs:812-815, 1165-1181).  One video.
__global__ void slot_rows_kernel(LinkInput in, LinkOutput out, const int64_t* __restrict__ row_off,
                                 int64_t* __restrict__ particle, int64_t* __restrict__ row_dur) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= in.npoints) return;
    const int g = (int)(p / in.slot_stride);
    const int64_t j = p - (int64_t)g * in.slot_stride;
    if (j >= (int64_t)in.gcount[g]) return;
    const int64_t row = row_off[g] + j;
    const int64_t id = (int64_t)(float)out.ids[p];
    particle[row] = id;
    if ((uint64_t)id >= (uint64_t)out.counter[0]) {
        atomicOr(out.flags, kFlagScratch);
        row_dur[row] = -1;
        return;
    }
    row_dur[row] = id_duration(out, id);
}

// --------------------------------------------------------------- launchers
cudaError_t link_sort_groups(const LinkInput& in, uint32_t* srt, uint8_t* scratch, size_t scratch_per_group,
                             int max_group, cudaStream_t st) {
    (void)max_group;
    if (in.ngroups == 0) return cudaSuccess;
    sort_groups_kernel<<<in.ngroups, kLinkThreads, 0, st>>>(in, srt, (uint64_t*)scratch, scratch_per_group / 8);
    return cudaGetLastError();
}

cudaError_t link_cells(const LinkInput& in, float4* rec, int32_t* cell_off, float4* geo, int g0, int g1,
                       cudaStream_t st) {
    if (g1 <= g0) return cudaSuccess;
    link_cells_kernel<<<g1 - g0, kCellThreads, 0, st>>>(in, g0, rec, cell_off, geo);
    return cudaGetLastError();
}

cudaError_t link_count_lists(const LinkInput& in, const uint32_t* srt, int64_t* f_cnt, int64_t* b_cnt,
                             cudaStream_t st) {
    LinkLists L;
    L.srt = (uint32_t*)srt;
    return link_count_lists_range(in, L, in.npoints, f_cnt, b_cnt, nullptr, st);
}

cudaError_t link_count_lists_range(const LinkInput& in, const LinkLists& L, int64_t p1, int64_t* f_cnt,
                                   int64_t* b_cnt, uint32_t* flags, cudaStream_t st) {
    const int64_t p0 = L.pbase;
    if (p1 <= p0) return cudaSuccess;
    lists_kernel<0><<<(unsigned)((p1 - p0 + 255) / 256), 256, 0, st>>>(in, L, f_cnt, b_cnt, p0, p1, flags);
    return cudaGetLastError();
}

cudaError_t link_fill_lists(const LinkInput& in, const LinkLists& L, cudaStream_t st) {
    return link_fill_lists_range(in, L, in.npoints, nullptr, st);
}

cudaError_t link_fill_lists_range(const LinkInput& in, const LinkLists& L, int64_t p1, uint32_t* flags,
                                  cudaStream_t st) {
    const int64_t p0 = L.pbase;
    if (p1 <= p0) return cudaSuccess;
    if ((L.f_cap >= 0 || L.b_cap >= 0) && !flags) return cudaErrorInvalidValue;
    lists_kernel<1><<<(unsigned)((p1 - p0 + 255) / 256), 256, 0, st>>>(in, L, nullptr, nullptr, p0, p1, flags);
    return cudaGetLastError();
}

cudaError_t link_run(const LinkInput& in, const LinkLists& L, const LinkScratch& S, const LinkOutput& out,
                     cudaStream_t st) {
    return link_run_window(in, L, S, out, LinkWindow(), st);
}

cudaError_t link_run_window(const LinkInput& in, const LinkLists& L, const LinkScratch& S, const LinkOutput& out,
                            const LinkWindow& w, cudaStream_t st) {
    if (in.nvideos == 0) return cudaSuccess;
    if (w.g0 >= 0 && (in.nvideos != 1 || !w.state)) return cudaErrorInvalidValue;
    // narrow offsets when the forward lists hold fewer than 2^31 entries
    const int64_t fmax = L.f_cap >= 0 ? L.f_cap : L.f_entries;
    if (fmax >= 0 && fmax < (int64_t)INT32_MAX) {
        constexpr size_t bytes = link_smem_bytes<int32_t>();
        cudaFuncSetAttribute(link_video_kernel<int32_t>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        link_video_kernel<int32_t><<<in.nvideos, kLinkThreads, bytes, st>>>(in, L, S, out, w);
    } else {
        constexpr size_t bytes = link_smem_bytes<int64_t>();
        cudaFuncSetAttribute(link_video_kernel<int64_t>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        link_video_kernel<int64_t><<<in.nvideos, kLinkThreads, bytes, st>>>(in, L, S, out, w);
    }
    return cudaGetLastError();
}

size_t link_segment_bytes(int32_t max_group, int64_t max_edges, int64_t npoints, int32_t memory) {
    return make_lay(max_group, max_edges, npoints, memory, true).total;
}

cudaError_t link_run_segments(const LinkInput& in, const LinkLists& L, const LinkScratch& S, const LinkOutput& out,
                              const LinkWindow& w, const LinkSegs& q, int64_t p0, int64_t p1, cudaStream_t st) {
    if (in.nvideos == 0) return cudaSuccess;
    if (w.g0 >= 0 && (in.nvideos != 1 || !w.state)) return cudaErrorInvalidValue;
    if (in.memory > kRingSmem || q.len < in.memory + 2 || q.prefix < 1 || q.max_segs < 1) return cudaErrorInvalidValue;
    const dim3 grid(q.max_segs, in.nvideos);
    const int64_t fmax = L.f_cap >= 0 ? L.f_cap : L.f_entries;
    if (fmax >= 0 && fmax < (int64_t)INT32_MAX) {
        constexpr size_t bytes = link_smem_bytes<int32_t>();
        cudaFuncSetAttribute(link_segments_kernel<int32_t>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        link_segments_kernel<int32_t><<<grid, kSegThreads, bytes, st>>>(in, L, S, out, w, q);
    } else {
        constexpr size_t bytes = link_smem_bytes<int64_t>();
        cudaFuncSetAttribute(link_segments_kernel<int64_t>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        link_segments_kernel<int64_t><<<grid, kSegThreads, bytes, st>>>(in, L, S, out, w, q);
    }
    if (p1 > p0)
        segment_ids_kernel<<<(unsigned)((p1 - p0 + 255) / 256), 256, 0, st>>>(in, S, out, w, q, p0, p1);
    return cudaGetLastError();
}

cudaError_t link_durations(const LinkInput& in, const LinkOutput& out, int64_t* row_dur, cudaStream_t st) {
    if (in.npoints == 0) return cudaSuccess;
    durations_kernel<<<(unsigned)((in.npoints + 255) / 256), 256, 0, st>>>(in, out, row_dur);
    return cudaGetLastError();
}

cudaError_t link_slot_rows(const LinkInput& in, const LinkOutput& out, const int64_t* row_off, int64_t* particle,
                           int64_t* row_dur, cudaStream_t st) {
    if (in.npoints == 0) return cudaSuccess;
    if (!in.slot_stride || in.nvideos != 1) return cudaErrorInvalidValue;
    slot_rows_kernel<<<(unsigned)((in.npoints + 255) / 256), 256, 0, st>>>(in, out, row_off, particle, row_dur);
    return cudaGetLastError();
}

}  // namespace gt
