// sort.cu -- voxel hash, counting sort and voxel table.
//
// Replaces the host-side voxel organisation of the reference
// (sim/src/sph/strategies/voxel_sph_strategy.py:65-107: GPU hash, copy to the
// host, numpy structured sort by (voxel_id, particle_id), Python loop building
// voxel_begin) with four device passes:
//   1. hash: voxel id per particle + atomic histogram (slot = arrival rank;
//      one atomic per run of lanes in the same voxel);
//   2. scan: exclusive prefix of the histogram = voxel_start (one pass);
//   3. scatter: particle id of each particle to voxel_start + slot;
//   4. rank-gather: each particle's final slot = voxel_start + number of
//      members of its voxel with a smaller particle id; the state is gathered
//      into that slot.  The result is the reference's (voxel, particle id)
//      order exactly, independent of atomic arrival order and of the input
//      order of the state.
// Voxels with more than kBigVoxel members (dense clusters, the overflow bucket
// of non-finite particles) have their member ids sorted between 3 and 4, by a
// quarter of a block each or a whole one, and the rank is a binary search, so
// the pass stays O(n log n) however the particles cluster.
#include <algorithm>
#include <climits>

#include "sphgb_internal.cuh"

namespace sphgb {

namespace {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 16;
constexpr int kScanTile = kScanThreads * kScanItems;  // 4096 voxels per tile

__device__ __forceinline__ int warp_incl_scan(int v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

__global__ void __launch_bounds__(512)
k_hash_count(const SceneDev* __restrict__ scenes, const int32_t* __restrict__ pbegin, int n_scenes,
             int i0, int i1, const float4* __restrict__ pos, int32_t* __restrict__ cell,
             int32_t* __restrict__ slot, int32_t* __restrict__ vcount) {
    const int s = grid_wait(i0 + (int)(blockIdx.x * blockDim.x + threadIdx.x));
    const int lane = threadIdx.x & 31;
    const bool valid = s < i1;
    int vid = -1;
    if (valid) {
        const SceneDev& sc = scenes[scene_of(s, pbegin, n_scenes)];
        const float4 p = __ldg(pos + s);
        if (finite3(p)) {
            const int vx = voxel_coord(p.x, sc.vs[0], sc.dims[0]);
            const int vy = voxel_coord(p.y, sc.vs[1], sc.dims[1]);
            const int vz = voxel_coord(p.z, sc.vs[2], sc.dims[2]);
            vid = sc.v_begin + voxel_index(vx, vy, vz, sc.tiled, sc.dims[0], sc.dims[1], sc.nt0, sc.nt1);
            cell[s] = vid;
        } else {
            vid = sc.v_begin + sc.v_count;   // overflow bucket
            cell[s] = ~vid;                  // negative: overflow bucket (no pid order needed)
        }
    }
    // Lanes of a run with the same voxel (sorted input holds whole voxels in
    // consecutive slots) take consecutive slots with one atomic by the run's
    // first lane.  Every lane of the warp takes part, in range or not.
    const unsigned full = 0xffffffffu;
    const int prev = __shfl_up_sync(full, vid, 1);
    const unsigned heads = __ballot_sync(full, !valid || lane == 0 || prev != vid);
    const unsigned le = (2u << lane) - 1u;
    const int leader = 31 - __clz(heads & le);
    int base = 0;
    if (valid && leader == lane) {
        const unsigned above = heads & ~le;
        const int next = above ? __ffs(above) - 1 : 32;
        base = atomicAdd(vcount + vid, next - lane);
    }
    base = __shfl_sync(full, base, leader);
    if (valid) slot[s] = base + (lane - leader);
}

// ---- scan ------------------------------------------------------------------
// One pass: a block scans its tile, publishes the tile's sum, adds up what the
// tiles before it have published, and publishes the sum up to its end
// (decoupled look-back: Merrill and Garland, NVR-2016-002).  A word of status
// holds a state and a value together: nothing else has to be ordered.  A tile
// that has published nothing after kScanPolls looks is not waited for: the
// warp adds up its counts itself, so the pass ends in whatever order the
// blocks run.  Against a reduction and a scan kernel, one launch less: the scan
// stage of 50k voxels 11.5 -> 8.4 us, of 2.5 M 20 -> 15.
constexpr unsigned long long kScanSum = 1ull << 32, kScanPrefix = 2ull << 32;
constexpr int kScanPolls = 256;

// sum of the counts of one tile, over a warp
__device__ __forceinline__ int tile_sum(const int32_t* __restrict__ vcount, int tile, int v_total) {
    const int lane = threadIdx.x & 31;
    const int k1 = min(v_total, (tile + 1) * kScanTile);
    int sum = 0;
    for (int k = tile * kScanTile + lane; k < k1; k += 32) sum += vcount[k];
    return __reduce_add_sync(0xffffffffu, sum);
}

// exclusive prefix of tile `tile` (the first warp of its block)
__device__ __forceinline__ int look_back(const int32_t* __restrict__ vcount, int v_total, int tile,
                                         const volatile unsigned long long* status) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    int before = 0;
    for (int last = tile - 1; last >= 0; last -= 32) {
        const int j = last - lane;          // lane 0: the nearest tile
        unsigned long long w = kScanPrefix; // before the first tile: nothing
        if (j >= 0) {
            w = status[j];
            for (int k = 0; w == 0 && k < kScanPolls; ++k) w = status[j];
        }
        for (unsigned late = __ballot_sync(full, w == 0); late; late &= late - 1) {
            const int l = __ffs(late) - 1;
            const int sum = tile_sum(vcount, last - l, v_total);
            if (lane == l) w = kScanSum | (unsigned)sum;
        }
        const unsigned ends = __ballot_sync(full, (w & kScanPrefix) != 0);
        const int stop = ends ? __ffs(ends) - 1 : 31;
        before += __reduce_add_sync(full, lane <= stop ? (int)(unsigned)w : 0);
        if (ends) break;
    }
    return before;
}

__global__ void __launch_bounds__(kScanThreads)
k_scan(const int32_t* __restrict__ vcount, int v_total, unsigned long long* status,
       int32_t* __restrict__ vstart, int4* __restrict__ next_counts, int next_quads) {
    __shared__ int s_before, s_warp[kScanThreads / 32];
    const int tile = grid_wait((int)blockIdx.x);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    // A warp's part of the tile in rows of 128, four entries per lane in each: whole
    // lines per access, where a lane's 16 entries in a row wrote half sectors, and
    // one barrier instead of two (699,220 particles in 48 boxes, 2.5 M entries:
    // stage 15.1 -> 13.3 us; step of 8,192 particles 26.0 -> 25.2).
    const int base = tile * kScanTile + wid * (32 * kScanItems) + 4 * lane;
    constexpr int kRows = kScanItems / 4;
    int4 v[kRows];
    const bool full = (tile + 1) * kScanTile <= v_total;
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
        const int k = base + 128 * i;
        if (full) {
            v[i] = __ldg(reinterpret_cast<const int4*>(vcount + k));
        } else {
            v[i].x = k < v_total ? __ldg(vcount + k) : 0;
            v[i].y = k + 1 < v_total ? __ldg(vcount + k + 1) : 0;
            v[i].z = k + 2 < v_total ? __ldg(vcount + k + 2) : 0;
            v[i].w = k + 3 < v_total ? __ldg(vcount + k + 3) : 0;
        }
    }
    int excl[kRows], in_warp = 0;
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
        const int sum = v[i].x + v[i].y + v[i].z + v[i].w;
        const int incl = warp_incl_scan(sum);
        excl[i] = in_warp + incl - sum;
        in_warp += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) s_warp[wid] = in_warp;
    __syncthreads();
    int before_warp = 0, total = 0;
#pragma unroll
    for (int w = 0; w < kScanThreads / 32; ++w) {
        const int t = s_warp[w];
        before_warp += w < wid ? t : 0;
        total += t;
    }
    if (threadIdx.x < 32) {
        volatile unsigned long long* mine = status + tile;
        if (threadIdx.x == 0) *mine = (tile ? kScanSum : kScanPrefix) | (unsigned)total;
        if (tile) {
            const int before = look_back(vcount, v_total, tile, status);
            if (threadIdx.x == 0) {
                *mine = kScanPrefix | (unsigned)(before + total);
                s_before = before;
            }
        } else if (threadIdx.x == 0) {
            s_before = 0;
        }
    }
    __syncthreads();
    const int off = before_warp + s_before;
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
        const int k = base + 128 * i;
        int4 o;
        o.x = off + excl[i];
        o.y = o.x + v[i].x;
        o.z = o.y + v[i].y;
        o.w = o.z + v[i].z;
        if (full) {
            *reinterpret_cast<int4*>(vstart + k) = o;
        } else {
            if (k < v_total) vstart[k] = o.x;
            if (k + 1 < v_total) vstart[k + 1] = o.y;
            if (k + 2 < v_total) vstart[k + 2] = o.z;
            if (k + 3 < v_total) vstart[k + 3] = o.w;
        }
    }
    // the next step's counters, status words and counts
    for (int k = blockIdx.x * kScanThreads + threadIdx.x; k < next_quads; k += gridDim.x * kScanThreads)
        next_counts[k] = make_int4(0, 0, 0, 0);
}

__global__ void __launch_bounds__(512)
k_scatter(int n, const int32_t* __restrict__ cell, const int32_t* __restrict__ slot,
          const int32_t* __restrict__ pid, const int32_t* __restrict__ vstart,
          const int32_t* __restrict__ vcount, int32_t* __restrict__ tmp_pid,
          int32_t* __restrict__ big_list, int32_t* __restrict__ big_count, int big_voxel) {
    const int s = grid_wait((int)(blockIdx.x * blockDim.x + threadIdx.x));
    if (s >= n) return;
    const int code = cell[s];
    const int vid = code < 0 ? ~code : code;
    const int sl = slot[s];
    tmp_pid[__ldg(vstart + vid) + sl] = pid[s];
    // overflow buckets (non-finite particles, never walked) keep arrival order
    if (code >= 0 && sl == 0 && __ldg(vcount + vid) > big_voxel)
        big_list[atomicAdd(big_count, 1)] = vid;
}

// One block per big voxel (grid-stride over the list): sorts the voxel's
// member ids ascending with a bitonic network whose comparators all put the
// smaller value at the lower index, so the segment is padded to a power of
// two implicitly (comparators reaching past the end are no-ops).  Segments up
// to kSmemSort ids are sorted in shared memory, longer ones in tiles of that
// size with the long comparators in global memory.
constexpr int kSortThreads = 1024;
constexpr int kSmemSort = 8192;

__device__ __forceinline__ void bitonic_pass(int32_t* a, int c, int n2, int k, int j) {
    const int half = n2 >> 1;
    for (int t = threadIdx.x; t < half; t += kSortThreads) {
        // j is a power of two: i = (t / j) 2 j + t % j.  The first step of a
        // merge mirrors within the k-block, the others are half-cleaners.
        const int i = ((t & ~(j - 1)) << 1) | (t & (j - 1));
        const int p = j == (k >> 1) ? i ^ (k - 1) : i + j;
        if (p < c) {
            const int32_t x = a[i], y = a[p];
            if (y < x) { a[i] = y; a[p] = x; }
        }
    }
}

// Segments up to kRankSort ids take a quarter of a block each and no sorting
// network: every id counts the smaller ones, from shared memory four at a time,
// all threads reading the same quad.  Equal ids (a caller's mistake) count by
// place, so the segment is sorted whatever the ids are: the rank-gather's binary
// search ends inside the voxel only in a sorted one.  A network of 1024
// threads per voxel spends its time in barriers (36 for 133 ids): the 4,000
// voxels of ~133 particles of the 262,144-particle pipe took 86 us, 13 us this
// way.  Beyond 512 ids the counting grows past the network (the pipe's later
// steps, voxels of 600 to 3,000: the sort 74 us with a limit of 1024, 49 with 512).
constexpr int kRankSort = 512;
constexpr int kQuarter = kSortThreads / 4;

__device__ __forceinline__ void quarter_sync(int quarter) {
    asm volatile("bar.sync %0, %1;" ::"r"(quarter + 1), "n"(kQuarter) : "memory");
}

__global__ void __launch_bounds__(kSortThreads)
k_sort_big(const int32_t* __restrict__ big_list, const int32_t* __restrict__ big_count,
           const int32_t* __restrict__ vstart, const int32_t* __restrict__ vcount,
           int32_t* __restrict__ tmp_pid) {
    __shared__ alignas(16) int32_t sm[kSmemSort];
    const int nb = *grid_wait(big_count);
    // most steps: nothing to do (51,911 particles: step 47.4 us through the barrier
    // below, 45.6 so)
    if (nb == 0) return;
    const int quarter = threadIdx.x / kQuarter, t = threadIdx.x % kQuarter;
    int32_t* sq = sm + quarter * kRankSort;
    for (int b = blockIdx.x * 4 + quarter; b < nb; b += gridDim.x * 4) {
        const int vid = big_list[b];
        const int st = vstart[vid], c = vcount[vid];
        if (c > kRankSort) continue;
        const int c4 = (c + 3) & ~3;
        for (int i = t; i < c4; i += kQuarter) sq[i] = i < c ? tmp_pid[st + i] : INT_MAX;
        quarter_sync(quarter);
        for (int i = t; i < c; i += kQuarter) {
            const int32_t p = sq[i];
            // equal ids keep their order: those before the warp's own 32 count, and
            // those of lower lanes
            const int own = i & ~31;
            const unsigned live = c - own >= 32 ? 0xffffffffu : (1u << (c - own)) - 1u;
            int r = __popc(__match_any_sync(live, p) & ((1u << (i & 31)) - 1u));
            int k = 0;
            for (; k < own; k += 4) {
                const int4 q = *reinterpret_cast<const int4*>(sq + k);
                r += (q.x <= p) + (q.y <= p) + (q.z <= p) + (q.w <= p);
            }
            for (; k < c4; k += 4) {
                const int4 q = *reinterpret_cast<const int4*>(sq + k);
                r += (q.x < p) + (q.y < p) + (q.z < p) + (q.w < p);
            }
            tmp_pid[st + r] = p;
        }
        quarter_sync(quarter);
    }
    // the longer ones, a whole block each (other voxels than the quarters': four
    // long ones of one block would wait for one another)
    bool any_long = false;
    for (int b = blockIdx.x + threadIdx.x * gridDim.x; b < nb; b += kSortThreads * gridDim.x)
        any_long |= vcount[big_list[b]] > kRankSort;
    if (!__syncthreads_or(any_long)) return;
    for (int b = blockIdx.x; b < nb; b += gridDim.x) {
        const int vid = big_list[b];
        const int st = vstart[vid], c = vcount[vid];
        if (c <= kRankSort) continue;
        int n2 = 1;
        while (n2 < c) n2 <<= 1;
        // A network's blocks of up to kSmemSort ids stay inside one aligned
        // tile, so a tile runs all its steps in shared memory, and only the
        // comparators that reach further work in global memory: 15 of the 171
        // passes over 262,144 ids.
        int32_t* a = tmp_pid + st;
        auto in_tiles = [&](int k0, int k1, int j_top) {
            for (int base = 0; base < c; base += kSmemSort) {
                const int m = min(kSmemSort, c - base);
                for (int i = threadIdx.x; i < m; i += kSortThreads) sm[i] = a[base + i];
                __syncthreads();
                for (int k = k0; k <= k1; k <<= 1)
                    for (int j = min(k >> 1, j_top); j > 0; j >>= 1) {
                        bitonic_pass(sm, m, min(n2, kSmemSort), k, j);
                        __syncthreads();
                    }
                for (int i = threadIdx.x; i < m; i += kSortThreads) a[base + i] = sm[i];
                __syncthreads();
            }
        };
        in_tiles(2, min(n2, kSmemSort), kSmemSort);
        for (int k = 2 * kSmemSort; k <= n2; k <<= 1) {
            for (int j = k >> 1; j >= kSmemSort; j >>= 1) {
                bitonic_pass(a, c, n2, k, j);
                __syncthreads();
            }
            in_tiles(k, k, kSmemSort / 2);
        }
    }
}

// kRows64: pipe scenes, with FP64 position rows to move too.  kDense: tasks of
// dense voxels have a list of their own.
template <bool kRows64, bool kDense>
__global__ void __launch_bounds__(512)
k_rank_gather(int n, const int32_t* __restrict__ cell, const int32_t* __restrict__ pid,
              const int32_t* __restrict__ tmp_pid, const int32_t* __restrict__ vstart,
              const int32_t* __restrict__ vcount, const float4* __restrict__ pos,
              const float4* __restrict__ vel, const double* __restrict__ pos64,
              float4* __restrict__ pos_out, float4* __restrict__ vel_out,
              int32_t* __restrict__ pid_out, double* __restrict__ pos64_out,
              TaskLists tasks, int big_voxel,
              const int32_t* __restrict__ slot, const int32_t* __restrict__ pbegin, int n_scenes,
              const int32_t* __restrict__ step_limit, const int32_t* __restrict__ scene_step) {
    const int s = grid_wait((int)(blockIdx.x * blockDim.x + threadIdx.x));
    if (s >= n) return;
    if (step_limit && scene_frozen(step_limit, scene_step, scene_of(s, pbegin, n_scenes))) {
        // frozen scene: every particle keeps its slot, no density task
        pid_out[s] = pid[s];
        pos_out[s] = __ldg(pos + s);
        if (vel) vel_out[s] = __ldg(vel + s);
        if (kRows64) {
            pos64_out[3 * s + 0] = pos64[3 * s + 0];
            pos64_out[3 * s + 1] = pos64[3 * s + 1];
            pos64_out[3 * s + 2] = pos64[3 * s + 2];
        }
        return;
    }
    const int code = cell[s];
    const int vid = code < 0 ? ~code : code;
    const int p = pid[s];
    // The chain from the cell to the rank is most of a small scene's pass: the
    // rows are loaded beside it, and the ids two quads at a time (8,192 particles:
    // step 27.1 -> 26.7 us, 699,220 in 48 boxes: pass 23.4 -> 22.7).  Not in pipe
    // scenes, whose threads have the FP64 rows to move too (pass 33 -> 36 us).
    float4 row = make_float4(0.f, 0.f, 0.f, 0.f), vrow = row;
    if (!kRows64) {
        row = __ldg(pos + s);
        if (vel) vrow = __ldg(vel + s);
    }
    const int st = __ldg(vstart + vid);
    const int c = __ldg(vcount + vid);
    int r = 0;
    if (code < 0) {
        r = slot[s];                    // overflow bucket: arrival order, no pid order
    } else if (c <= big_voxel) {
        // the voxel's ids four per load from the aligned quad at or before st;
        // entries outside [st, st + c) are masked (tmp_pid is 16-byte aligned
        // and padded by 4 entries, so the last quad stays inside it; a second quad
        // past the end is not loaded)
        const int e = st + c;
#pragma unroll 1
        for (int k = st & ~3; k < e; k += 8) {
            const int4 q = __ldg(reinterpret_cast<const int4*>(tmp_pid + k));
            const int k2 = k + 4 < e ? k + 4 : k;
            const int4 q2 = __ldg(reinterpret_cast<const int4*>(tmp_pid + k2));
            r += (k >= st && q.x < p) + (k + 1 >= st && k + 1 < e && q.y < p) +
                 (k + 2 >= st && k + 2 < e && q.z < p) + (k + 3 < e && q.w < p);
            r += (k + 4 < e && q2.x < p) + (k + 5 < e && q2.y < p) + (k + 6 < e && q2.z < p) +
                 (k + 7 < e && q2.w < p);
        }
    } else {                            // sorted by k_sort_big: lower bound of p
        int lo = 0, hi = c;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (__ldg(tmp_pid + st + mid) < p) lo = mid + 1; else hi = mid;
        }
        r = lo;
    }
    const int d = st + r;
    if (tasks.list && (r % kTaskRun) == 0) {
        int first = vid;
        bool mine = true;
        if (c < tasks.pair_max && code >= 0) {
            const int other = __ldg(vcount + (vid ^ 16));
            if (other > 0 && c + other <= tasks.pair_max) {
                first = ~vid;
                mine = !(vid & 16);       // the even voxel's first particle lists the pair
            }
        }
        if (!mine) {
        } else if (kDense && c >= tasks.dense_from &&
                   (!tasks.scenes ||
                    tasks.scenes[scene_of(s, pbegin, n_scenes)].cap <= kListCap))
            tasks.dense_last[-atomicAdd(tasks.dense_count, 1)] = make_int2(vid, d);
        else
            tasks.list[atomicAdd(tasks.count, 1)] = make_int2(first, d);
    }
    pid_out[d] = p;
    if (kRows64) {
        row = __ldg(pos + s);
        if (vel) vrow = __ldg(vel + s);
    }
    pos_out[d] = row;
    if (vel) vel_out[d] = vrow;             // null: velocities gathered later
    if (kRows64) {
        pos64_out[3 * d + 0] = pos64[3 * s + 0];
        pos64_out[3 * d + 1] = pos64[3 * s + 1];
        pos64_out[3 * d + 2] = pos64[3 * s + 2];
    }
}

}  // namespace

int scan_tiles(int v_total) { return (v_total + kScanTile - 1) / kScanTile; }

cudaError_t launch_hash_count(const Launch& L, const float4* pos, int32_t* cell, int32_t* slot,
                              int32_t* vcount, int i0, int i1) {
    if (i1 < 0) i1 = L.n;
    if (i0 < 0 || i1 > L.n || i0 > i1) return cudaErrorInvalidValue;
    if (i1 == i0) return cudaSuccess;
    const int b = L.sort_block;
    return launch_chained(k_hash_count, (i1 - i0 + b - 1) / b, b, L, L.scenes, L.pbegin,
                          L.n_scenes, i0, i1, pos, cell, slot, vcount);
}

cudaError_t launch_scan(const Launch& L, const int32_t* vcount, int32_t* vstart,
                        unsigned long long* status, int n_tiles, int32_t* next_counts,
                        size_t next_ints) {
    if (L.v_total == 0) return cudaSuccess;
    return launch_chained(k_scan, n_tiles, kScanThreads, L, vcount, L.v_total, status, vstart,
                          reinterpret_cast<int4*>(next_counts),
                          next_counts ? (int)(next_ints / 4) : 0);
}

cudaError_t launch_scatter(const Launch& L, const int32_t* cell, const int32_t* slot,
                           const int32_t* pid, const int32_t* vstart, const int32_t* vcount,
                           int32_t* tmp_pid, int32_t* big_list, int32_t* big_count) {
    if (L.n == 0) return cudaSuccess;
    const int b = L.sort_block;
    return launch_chained(k_scatter, (L.n + b - 1) / b, b, L, L.n, cell, slot, pid, vstart,
                          vcount, tmp_pid, big_list, big_count, L.big_voxel);
}

cudaError_t launch_sort_big(const Launch& L, const int32_t* big_list, const int32_t* big_count,
                            const int32_t* vstart, const int32_t* vcount, int32_t* tmp_pid) {
    if (L.n == 0) return cudaSuccess;
    // two blocks (eight quarters) per SM, no more quarters than there can be
    // big voxels; idle blocks exit at once
    const int most = (L.n / L.big_voxel + 4) / 4;
    return launch_chained(k_sort_big, std::min(most, device_sm_count() * 2), kSortThreads, L,
                          big_list, big_count, vstart, vcount, tmp_pid);
}

cudaError_t launch_rank_gather(const Launch& L, const int32_t* cell, const int32_t* slot,
                               const int32_t* pid, const int32_t* tmp_pid, const int32_t* vstart,
                               const int32_t* vcount, const float4* pos, const float4* vel,
                               const double* pos64, float4* pos_out, float4* vel_out,
                               int32_t* pid_out, double* pos64_out, TaskLists tasks) {
    if (L.n == 0) return cudaSuccess;
    const int b = L.sort_block;
    // k_density_tc is chained to this one, its blocks fill the shared memory, and an
    // SM is not set up anew while it has blocks: this pass runs with the density
    // pass's set-up (17,280 particles: step 35.8 -> 34.5 us, 51,911: 49.9
    // -> 48.9).  A density pass that is not chained is as fast there but loses 1 to
    // 3 us in a single step.  More particles than resident threads use what the
    // blocks before left in L1 (4,194,304: pass 97 us, 120 with little L1; a dense
    // pipe's 262,144, before k_density_wc, 23 and 33).
    Launch next = L;
    if (tasks.tc_next && L.n <= 2048 * device_sm_count()) next.smem_share = 100;
    auto kernel = tasks.dense_last ? (pos64 ? k_rank_gather<true, true> : k_rank_gather<false, true>)
                                   : (pos64 ? k_rank_gather<true, false> : k_rank_gather<false, false>);
    return launch_chained(kernel, (L.n + b - 1) / b, b, next, L.n, cell, pid, tmp_pid, vstart,
                          vcount, pos, vel, pos64, pos_out, vel_out, pid_out, pos64_out, tasks,
                          L.big_voxel, slot, L.pbegin, L.n_scenes, L.step_limit, L.scene_step);
}

}  // namespace sphgb
