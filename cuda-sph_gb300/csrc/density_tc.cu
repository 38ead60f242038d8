// density_tc.cu -- the density pass of the step for sparse scenes and scenes
// without a neighbour cap: neighbour decisions on the tensor cores.  Dense
// scenes run k_density_wc (walk.cu), whose homes skip voxels one by one.
#include <algorithm>
#include <climits>
#include <cuda_fp16.h>

#include "sphgb_internal.cuh"

namespace sphgb {

namespace {

// Warp-cooperative density pass of the step.  One warp per task: up to
// kTaskRun particles ("homes") of one voxel, or of two that are neighbours in z
// (tasks listed by the rank-gather, see TaskLists).  The 27 walk voxels of that
// voxel, or the 36 of the two, are laid end to end in walk order and taken
// in chunks of kTcChunk candidates.  Per chunk:
//
// Phase 1 decides every (home, candidate) pair into one bit, 32 candidates (a
// group) per word.  The squared distances of 16 homes to 8 candidates are a
// contraction, |u_j|^2 - 2 u_i.u_j + |u_i|^2 with u the position relative to
// the voxel's centre in voxel sizes, so it runs as one mma.sync m16n8k16 on
// FP16 pairs (each coordinate as a high and a low half, 22 bits) with FP32
// accumulation: four instructions test 512 pairs, and the accumulator started
// at |u_i|^2 - h^2 leaves the decision in the sign bit.  The result is within
// kTcTol of d^2 - h^2; a home with a pair closer to the threshold than that
// has its group decided again with the walk's FP32 arithmetic and FP64 guard
// band, as has a group with a particle far outside its voxel (clamped
// coordinates), so the decisions are the reference's, bit for bit.  Tasks of
// few homes (kTcBallot) test with FP32 ballots, which cost per home.  Groups
// run until every home is at its cap.  (The tcgen05 tiles start at 64 rows; the
// rows here are the at most 16 particles that share a candidate list.)
//
// Phase 2 walks each home's bits in order, two lanes per home (the two parts
// of the sum, see kSumSplit): neighbour slot into the list row, squared
// distance with the walk's FP32 arithmetic, density term, Kahan sum.  The sum
// is that of density_one, so both kernels give the same bits.
//
// What bounds it: instruction issue (70 % of the issue slots with 24 warps per
// SM) beside the L1 / shared-memory pipe (76 %).  A 4,194,304-particle box
// at 11 particles per voxel: 1.171 ms with the ballots and per-home ranking of
// k_density_wc, 0.940 ms here, 2765 against 2000 warp instructions per task of
// 10 homes (400 to set up, 100 per group of candidates for all homes, 760 in
// phase 2).  262,144 particles: 88 -> 71 us.  Measured and not kept: 32 warps per
// SM at 64 registers (1.09 ms: spills, 20 % more instructions), 16-bit list
// entries, one lane per (home, word) extracting the bits into lists and one
// lane per list entry for the terms (1.29 ms: dense words make the extraction
// as long as the longest), the next batch loaded during the decisions (1.24
// ms: spills), 1 or 3 groups per batch (1.10, 1.41).
constexpr int kTcWarps = 4;
constexpr int kTcGroups = 2;                 // groups of 32 candidates per batch
constexpr int kTcBatch = 32 * kTcGroups;
constexpr int kTcChunk = 320;                // candidates held in shared memory
constexpr int kTcWords = kTcChunk / 32;
// Walks longer than this pass over unreachable batches: two chunks and more.  At 320
// the masks cost more than they save (4,194,304-particle box 0.967 ms, 0.940 so);
// beyond 640, or never, within 1 % from 4 to 80 particles per voxel.
constexpr int kTcCullMin = 640;
// Tasks of at most this many homes test with ballots: 0.940 ms with 2 as with
// 4, 0.973 with 8.
constexpr int kTcBallot = 4;
// Bound on |computed - exact| of (d^2 - h^2) / vs^2 for candidates of |u|^2 <=
// kTcFar, homes of |u|^2 <= kTcHome and (h / vs)^2 <= kTcH2 (others are decided
// by ballots): every partial sum is below 9 + 2 sqrt(9 * 1.6) + 2 < 32.  The FP32
// rounding of u and |u|^2 gives 2^-17.4, the FP16 pairs 2^-17.4 over the products
// and |u|^2, 17 accumulations truncated at 2^-19 each 2^-14.9: 2^-14.4 = 5e-5
// together.  (PTX gives mma's FP32 accumulation at least single precision and
// leaves the rounding open: truncation of 24 bits is the worst it allows.)
constexpr float kTcTol = 1.0e-4f;
constexpr float kTcFar = 9.0f;    // |u|^2 within the walk: 3 * 1.5^2, pairs 2 * 1.5^2 + 2^2
constexpr float kTcHome = 1.6f;   // 3 * 0.5^2, pairs 2 * 0.5^2 + 1
constexpr float kTcH2 = 2.0f;
static_assert(kTcChunk % kTcBatch == 0, "a chunk is whole batches");
static_assert(kTaskRun == 16 && kTaskRun <= kSumSplit, "16 rows per mma, two lanes per home");

constexpr int kTcRow = kListCap + 4;           // rows apart by 4 banks, read as int4
constexpr int kTcMaskRow = kTcWords | 1;       // rows in different banks
struct alignas(16) TcShared {
    float4 cand[kTcChunk];             // x, y, z and the slot (int bits) of each candidate
    uint4 feat[kTcBatch];              // FP16 features of a batch, in ldmatrix order
    int32_t list[kTaskRun][kTcRow];    // neighbour slots in walk order
    uint32_t mask[kTaskRun][kTcMaskRow];   // accepted candidates: word q >> 5, q & 31 from the top bit
    uint32_t seg[kTcWords];       // chunk's places where a walk voxel starts, bit q & 31 of word q >> 5
    uint32_t reach1[16];          // see TcWalk
    int32_t off[36];              // first slot - first walk index of each non-empty walk voxel, by rank
};

__device__ __forceinline__ uint32_t half2_bits(float lo, float hi) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ float2 half2_floats(uint32_t b) {
    return __half22float2(*reinterpret_cast<const __half2*>(&b));
}
// u as high and low halves: (xh, yh), (zh, wh), (xl, yl), (zl, wl)
__device__ __forceinline__ uint4 split_halves(float x, float y, float z, float w) {
    uint4 f;
    f.x = half2_bits(x, y);
    f.y = half2_bits(z, w);
    const float2 a = half2_floats(f.x), b = half2_floats(f.y);
    f.z = half2_bits(x - a.x, y - a.y);
    f.w = half2_bits(z - b.x, w - b.y);
    return f;
}
// smallest of the three magnitudes, one instruction (sm_100)
__device__ __forceinline__ float min_abs3(float a, float b, float c) {
    float r;
    asm("min.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
// d = A b + c for 8 candidates; b0 and b1 are the same features, which A meets
// with the high halves of the homes' coefficients (k < 8) and the low ones
__device__ __forceinline__ void mma_16x8x16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0,
                                            uint32_t b1, const float (&c)[4]) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%10,%11,%12,%13};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c[0]), "f"(c[1]),
          "f"(c[2]), "f"(c[3]));
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&b)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3])
                 : "r"(addr)
                 : "memory");
}
// home i of the task (its lane's position), to every lane
__device__ __forceinline__ float4 home_of(const float4& pi, int i) {
    return make_float4(__shfl_sync(0xffffffffu, pi.x, i), __shfl_sync(0xffffffffu, pi.y, i),
                       __shfl_sync(0xffffffffu, pi.z, i), 0.0f);
}

// The scene's frame for one task: u = (p - o) * s
struct TcFrame {
    float ox, oy, oz, s;
};

// the exact decision of the 32 candidates of a group (one per lane) for home
// ph, the first candidate in the top bit
__device__ __forceinline__ unsigned group_mask(const float4& ph, const float4& pj, float h2_lo,
                                               float h2_hi, double h_d) {
    const float d2 = dist2(ph, pj);
    bool acc = d2 < h2_lo;
    if (!acc && d2 <= h2_hi) acc = within_exact(ph.x, ph.y, ph.z, pj.x, pj.y, pj.z, h_d);
    return __brev(__ballot_sync(0xffffffffu, acc));
}

// A task's walk as one lane holds it: lane l < 18 has the column l / 2 of the
// walk (x and y neighbours, in walk order) and two of its voxels in z, with
// the walk indices where they start and end.  reach0 and S.reach1 of home lane &
// 15 (long walks): bit l set when lane l's first or second voxel may hold a
// particle within h of it.
struct TcWalk {
    int p0, p1, end;
    unsigned reach0;
    __device__ __forceinline__ bool has0() const { return p1 > p0; }
    __device__ __forceinline__ bool has1() const { return end > p1; }
    // Sets S.seg's bits for the chunk at c0.  Candidate q of the walk lies in the
    // last non-empty walk voxel that starts at or before it, found by counting
    // the bits.
    __device__ __forceinline__ void mark(TcShared& S, int c0) const {
        const unsigned a = p0 - c0, b = p1 - c0;
        if (has0() && a < kTcChunk) atomicOr(&S.seg[a >> 5], 1u << (a & 31));
        if (has1() && b < kTcChunk) atomicOr(&S.seg[b >> 5], 1u << (b & 31));
    }
};

// Phase 1 for the candidates [c0, c1) of one task: writes S.cand and S.mask
// and returns the number of groups decided; T receives each home's accepted
// candidates (lanes i and 16 + i: home i), and (gh, Th) the last word with at
// most kSumSplit accepted candidates of the home before it, and how many of
// them are in the chunk.  Stops early once every home has `cap` (cnt: accepted
// before this chunk).  cull: batches that no home reaches are passed over.
__device__ __forceinline__ int tc_decide(TcShared& S, int& T, int& gh, int& Th, int cnt, int c_t,
                                         int cap, int c0, int c1, const TcWalk& W, bool cull,
                                         const uint32_t (&A)[4], const float (&C)[4], bool ballots,
                                         const TcFrame& F, const float4& pi,
                                         const float4* __restrict__ pos, int n, const SceneDev& sc) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int ih = lane & 15;
    const unsigned le = (2u << lane) - 1u;      // bits 0..lane
    // rank: the last non-empty walk voxel that starts before the group, taking bit
    // 0 of the chunk's first word for a start
    int rank = -1;
    if (c0 > 0) {
        if (lane < kTcWords) S.seg[lane] = lane == 0 ? 1u : 0u;
        rank += __popc(__ballot_sync(full, W.has0() && W.p0 <= c0)) +
                __popc(__ballot_sync(full, W.has1() && W.p1 <= c0)) - 1;
        __syncwarp();
        W.mark(S, c0);
        __syncwarp();
    }
    // Candidate l of a group is column n = 2 (l / 8) + l % 2 of mma t =
    // (l / 2) % 4, so that lane 4 r + q ends up with the decisions of home r
    // (and r + 8) on candidates 8 q .. 8 q + 7, byte 3 - q of the mask word.  The
    // features lie 8 rows per mma, rows swapped within them so that neither
    // the stores nor the ldmatrix meet a bank twice.  An ldmatrix takes the
    // rows of two mmas, each twice: the two k-halves of B.
    const int st_t = (lane >> 1) & 3, st_n = ((lane >> 3) << 1) | (lane & 1);
    uint4* f_store = S.feat + st_t * 8 + (st_n ^ (2 * st_t));
    const int ld_t = lane >> 4;
    const uint32_t f_load0 = smem_addr(S.feat + ld_t * 8 + ((lane & 7) ^ (2 * ld_t)));
    const uint32_t f_load1 = smem_addr(S.feat + (ld_t + 2) * 8 + ((lane & 7) ^ (2 * (ld_t + 2))));
    uint8_t* mbyte = reinterpret_cast<uint8_t*>(S.mask[lane >> 2]) + (3 - (lane & 3));
    int G = 0;
    T = gh = Th = 0;
    for (int b0 = c0; b0 < c1; b0 += kTcBatch, G += kTcGroups) {
        if (cull) {
            // walk voxels overlapping this batch: skipped when no home below
            // the cap reaches one (those voxels hold no accepted candidate)
            const unsigned s0 = __ballot_sync(full, W.has0() && W.p0 < b0 + kTcBatch && W.p1 > b0);
            const unsigned s1 = __ballot_sync(full, W.has1() && W.p1 < b0 + kTcBatch && W.end > b0);
            if (!__any_sync(full, ih < c_t && cnt + T < cap &&
                                      ((W.reach0 & s0) | (S.reach1[ih] & s1)) != 0u)) {
#pragma unroll
                for (int u = 0; u < kTcGroups; ++u) {
                    if (lane < kTaskRun) S.mask[ih][G + u] = 0u;
                    if (cnt + T <= kSumSplit) { gh = G + u; Th = T; }
                    rank += __popc(S.seg[G + u]);
                }
                __syncwarp();
                continue;
            }
        }
        // Past the end of the walk (the last batch) some particle stands in,
        // and its bits are cut off below.
        float4 pj[kTcGroups];
#pragma unroll
        for (int u = 0; u < kTcGroups; ++u) {
            const unsigned starts = S.seg[G + u];
            const int sj = min(b0 + 32 * u + lane + S.off[rank + __popc(starts & le)], n - 1);
            pj[u] = __ldg(pos + sj);
            pj[u].w = __int_as_float(sj);
            rank += __popc(starts);
        }
        // the bits of group u that are candidates
        auto valid = [&](int u) {
            const int v = c1 - b0 - 32 * u;
            return v >= 32 ? full : v <= 0 ? 0u : ~(full >> v);
        };
        const bool tail = b0 + kTcBatch > c1;
#pragma unroll
        for (int u = 0; u < kTcGroups; ++u) S.cand[b0 - c0 + 32 * u + lane] = pj[u];
        if (ballots) {
            const float h2_lo = sc.h2_lo, h2_hi = sc.h2_hi;
            for (int i = 0; i < c_t; ++i) {
                const float4 ph = home_of(pi, i);
#pragma unroll
                for (int u = 0; u < kTcGroups; ++u) {
                    const unsigned m = group_mask(ph, pj[u], h2_lo, h2_hi, sc.h_d) & valid(u);
                    if (lane == 0) S.mask[i][G + u] = m;
                }
            }
        } else {
            bool far = false;
#pragma unroll
            for (int u = 0; u < kTcGroups; ++u) {
                const float x = (pj[u].x - F.ox) * F.s, y = (pj[u].y - F.oy) * F.s,
                            z = (pj[u].z - F.oz) * F.s;
                const float c = x * x + y * y + z * z;
                // far from the voxel (its halves may overflow): the batch is decided again
                far |= !(c <= kTcFar) && b0 + 32 * u + lane < c1;
                f_store[32 * u] = split_halves(x, y, z, c);
            }
            const bool any_far = __any_sync(full, far);     // and the warp's stores are in
            __syncwarp();
#pragma unroll
            for (int u = 0; u < kTcGroups; ++u) {
                uint32_t b[8];
                ldmatrix_x4(reinterpret_cast<uint32_t(&)[4]>(b[0]), f_load0 + u * 32 * (uint32_t)sizeof(uint4));
                ldmatrix_x4(reinterpret_cast<uint32_t(&)[4]>(b[4]), f_load1 + u * 32 * (uint32_t)sizeof(uint4));
                unsigned m0 = 0, m1 = 0;
                float near0 = 1.0f, near1 = 1.0f;
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    float d[4];
                    mma_16x8x16(d, A, b[2 * t], b[2 * t + 1], C);
                    m0 = __funnelshift_l(__float_as_uint(d[0]), m0, 1);
                    m0 = __funnelshift_l(__float_as_uint(d[1]), m0, 1);
                    m1 = __funnelshift_l(__float_as_uint(d[2]), m1, 1);
                    m1 = __funnelshift_l(__float_as_uint(d[3]), m1, 1);
                    near0 = min_abs3(near0, d[0], d[1]);
                    near1 = min_abs3(near1, d[2], d[3]);
                }
                if (tail) {
                    const unsigned v = valid(u) >> (24 - 8 * (lane & 3));
                    m0 &= v;
                    m1 &= v;
                }
                mbyte[4 * (G + u)] = (uint8_t)m0;
                mbyte[4 * (G + u) + 8 * kTcMaskRow * (int)sizeof(uint32_t)] = (uint8_t)m1;
                if (__any_sync(full, near0 < kTcTol || near1 < kTcTol) || any_far) {
                    // rows (homes) to decide again: four flag bits per row
                    unsigned f0 = __ballot_sync(full, near0 < kTcTol || any_far);
                    unsigned f1 = __ballot_sync(full, near1 < kTcTol || any_far);
                    __syncwarp();
                    while (f0 | f1) {
                        const bool low = f0 != 0u;
                        const int bit = __ffs(low ? f0 : f1) - 1;
                        const int i = (bit >> 2) + (low ? 0 : 8);
                        if (low) f0 &= ~(15u << (bit & ~3)); else f1 &= ~(15u << (bit & ~3));
                        if (i >= c_t) continue;
                        const unsigned m = group_mask(home_of(pi, i), pj[u], sc.h2_lo, sc.h2_hi,
                                                      sc.h_d) & valid(u);
                        if (lane == 0) S.mask[i][G + u] = m;
                    }
                }
            }
        }
        __syncwarp();
#pragma unroll
        for (int u = 0; u < kTcGroups; ++u) {
            if (cnt + T <= kSumSplit) { gh = G + u; Th = T; }
            T += __popc(S.mask[ih][G + u]);
        }
        if (!__any_sync(full, ih < c_t && cnt + T < cap)) {
            G += kTcGroups;
            break;
        }
    }
    return G;
}

// A lane's place in the accepted bits of its home: the bits of a word still to
// visit, the word after it (loaded ahead), and the shared-memory addresses of
// the word's first candidate and of the word after `next`.
struct TcCursor {
    uint32_t w, next, cand, after;
    __device__ __forceinline__ TcCursor(const TcShared& S, int ih, int g, uint32_t w_) {
        w = w_;
        next = S.mask[ih][g + 1];
        cand = smem_addr(S.cand + 32 * g);
        after = smem_addr(&S.mask[ih][g + 2]);
    }
    // at the end of a word: on to the next one, without a branch
    __device__ __forceinline__ void advance_if_empty() {
        asm volatile("{\n\t.reg .pred p;\n\t"
                     "setp.eq.u32 p, %0, 0;\n\t"
                     "@p mov.b32 %0, %1;\n\t"
                     "@p add.u32 %2, %2, %4;\n\t"
                     "@p ld.shared.b32 %1, [%3];\n\t"
                     "@p add.u32 %3, %3, 4;\n\t}"
                     : "+r"(w), "+r"(next), "+r"(cand), "+r"(after)
                     : "n"(32 * sizeof(float4))
                     : "memory");
    }
};

// w without its first d bits (from the top; it has at least d)
__device__ __forceinline__ uint32_t drop_first(uint32_t w, int d) {
    int at = 0;      // the most leading places that hold at most d bits
#pragma unroll
    for (int s = 16; s > 0; s >>= 1)
        if (__popc(w & ~(0xffffffffu >> (at + s))) <= d) at += s;
    return w & (0xffffffffu >> at);
}

// Phase 2 for one lane: visits the next n accepted candidates of its home,
// adds their density terms and stores their slots from shared-memory address
// `row` on (kBound: below row_end only, and below over_end from `over` on),
// passing over the one at address `self`; returns where the row ends.
// The words hold at least n more bits: n counts bits of theirs.  A lane that
// meets an empty word lets a turn pass.
template <bool kBound>
__device__ __forceinline__ uint32_t tc_sum(TcCursor& C, int n, uint32_t row, uint32_t row_end,
                                           uint32_t self, const float4& pi, float inv_h2,
                                           Kahan& acc, int32_t* over = nullptr,
                                           uint32_t over_end = 0u) {
    while (n > 0) {
        C.advance_if_empty();
        // place of the first bit; -1 in an empty word, which is never the
        // chunk's first one, so that the read below stays inside S.cand
        int z;
        asm("bfind.shiftamt.u32 %0, %1;" : "=r"(z) : "r"(C.w));
        uint32_t bit;
        asm("shr.b32 %0, %1, %2;" : "=r"(bit) : "r"(0x80000000u), "r"(z));   // 0 past 31
        C.w ^= bit;
        const uint32_t at = C.cand + z * (int)sizeof(float4);
        float4 pj;
        asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];"
                     : "=f"(pj.x), "=f"(pj.y), "=f"(pj.z), "=f"(pj.w)
                     : "r"(at)
                     : "memory");
        const float u = __fmaf_rn(-dist2(pi, pj), inv_h2, 1.0f);
        Kahan a = acc;
        a.add(u * u * u);
        if (z >= 0) --n;
        if (z >= 0 && at != self) {
            acc = a;
            if (!kBound || row < row_end)
                asm volatile("st.shared.f32 [%0], %1;" ::"r"(row), "f"(pj.w) : "memory");
            if (kBound) {
                if (row < over_end) *over = __float_as_int(pj.w);
                ++over;
            }
            row += 4;
        }
    }
    return row;
}

// kLayout: 0 every scene's voxel table row-major, 1 every one tiled, 2 per scene.
// kUncapped: some scene's cap is beyond kListCap.
// kGather: the task's velocities too, from FP64 rows (vrows).
template <int kLayout, bool kUncapped, bool kGather>
__global__ void __launch_bounds__(kTcWarps * 32, 6)
k_density_tc(const SceneDev* __restrict__ scenes, const int32_t* __restrict__ pbegin,
             int n_scenes, int n, const float4* __restrict__ pos,
             const float4* __restrict__ vel, const int32_t* __restrict__ vstart,
             const int32_t* __restrict__ vcount, float* __restrict__ rho,
             float4* __restrict__ fin, NbrList nbr,
             const int2* __restrict__ tasks, const int32_t* __restrict__ task_count,
             int32_t* __restrict__ task_next, const int32_t* __restrict__ task_offset,
             VelRows vrows) {
    __shared__ TcShared sh[kTcWarps];
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    TcShared& S = sh[threadIdx.x >> 5];
    const unsigned lt = (1u << lane) - 1u;
    if (lane < kTcWords) S.seg[lane] = 0u;
    __syncwarp();
    int n_tasks = *grid_wait(task_count);
    if (nbr.veto && *after_wait(nbr.veto)) n_tasks = 0;
    if (task_offset) tasks += *after_wait(task_offset);   // one bucket of a bucketed task list
    // A warp's first task is its own number; each later one comes from a
    // counter (the cost of a task varies with its voxel's neighbourhood, and a
    // fixed share per warp left warps idle at the end of the pass, 15 % of its
    // time on the 4M box), taken while the task before it runs.
    const int n_warps = gridDim.x * kTcWarps;
    int next = blockIdx.x * kTcWarps + (threadIdx.x >> 5);
    for (;;) {
        const int t = __shfl_sync(full, next, 0);    // uniform, also to the compiler
        if (t >= n_tasks) break;
        const int2 task = after_wait(tasks)[t];
        if (lane == 0) next = n_warps + atomicAdd(task_next, 1);
        // a pair task (see TaskLists) has its first voxel's index complemented
        const bool pair = kLayout == 1 && !kGather && task.x < 0;
        const int vid = pair ? ~task.x : task.x, d0 = task.y;
        const SceneDev& sc = scenes[scene_of_warp(d0, pbegin, n_scenes)];
        const int local = vid - sc.v_begin;
        const int cap = sc.cap;
        // the walk voxels (voxel_kernels.py:46-61 order), from the table coords
        const int tiled = kLayout == 2 ? sc.tiled : kLayout;
        // index -> coordinates with the scene's multiply-shift reciprocals
        const Udiv q0{sc.div_m[0], sc.div_s[0]}, q1{sc.div_m[1], sc.div_s[1]};
        int vx, vy, vz;
        if (tiled) {
            const int tl = local >> 6, in = local & 63;
            const int r0 = q0.div(tl), r1 = q1.div(r0);
            vx = ((tl - r0 * sc.nt0) << 2) | (in & 3);
            vy = ((r0 - r1 * sc.nt1) << 2) | ((in >> 2) & 3);
            vz = (r1 << 2) | (in >> 4);
        } else {
            const int r0 = q0.div(local), r1 = q1.div(r0);
            vx = local - r0 * sc.dims[0];
            vy = r0 - r1 * sc.dims[1];
            vz = r1;
        }
        // 9 columns of 3 voxels in z, or of 4 for a pair: each home's own walk is
        // in order in them, and the voxel that is not in it lies a whole voxel
        // side away, so that its particles are beyond h
        TcWalk W{0, 0, 0, 0u};
        int wc0, wc1, st0, st1, id0, id1;
        {
            const int col = lane >> 1, half = lane & 1;
            const int nx = vx + col / 3 - 1, ny = vy + col % 3 - 1, nz = vz - 1 + 2 * half;
            const int w0 = sc.wdims[0], w1 = sc.wdims[1], w2 = sc.wdims[2];
            const bool in = lane < 18 && nx >= 0 && nx < w0 && ny >= 0 && ny < w1;
            const bool in0 = in && nz >= 0 && nz < w2, in1 = in && (half == 0 || pair) && nz + 1 < w2;
            id0 = in0 ? sc.v_begin + voxel_index(nx, ny, nz, tiled, w0, w1, sc.nt0, sc.nt1) : vid;
            id1 = in1 ? sc.v_begin + voxel_index(nx, ny, nz + 1, tiled, w0, w1, sc.nt0, sc.nt1) : vid;
            wc0 = __ldg(vcount + id0);
            wc1 = __ldg(vcount + id1);
            st0 = __ldg(vstart + id0);
            st1 = __ldg(vstart + id1);
            wc0 = in0 ? wc0 : 0;
            wc1 = in1 ? wc1 : 0;
        }
        // lanes i and 16 + i: home i, at slot s (loaded beside the counts that say
        // how many there are)
        const int ih = lane & 15;
        int s = d0 + ih;
        float4 pi = __ldg(pos + min(s, n - 1));
        // the task's particles: a run of its voxel, or all of the pair's two (the
        // second voxel is the first one of lane 9)
        const int vst = __ldg(vstart + vid), vc = __ldg(vcount + vid);
        const int st_b = __shfl_sync(full, st0, 9), c_b = __shfl_sync(full, wc0, 9);
        const int c_a = min(kTaskRun, vst + vc - d0);
        const int c_t = pair ? c_a + c_b : c_a;
        const bool upper = lane >= 16, home = lane < c_t;
        if (ih >= c_a) {
            s = st_b + ih - c_a;
            pi = make_float4(0.f, 0.f, 0.f, 0.f);
            if (ih < c_t) pi = __ldg(pos + s);
        }
        int incl = wc0 + wc1;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(full, incl, o);
            if (lane >= o) incl += v;
        }
        // candidates in the whole walk; none for the overflow entry, whose
        // particles (non-finite positions) have no neighbours
        const int M = local == sc.v_count ? 0 : __shfl_sync(full, incl, 17);
        // Candidate q (walk order) lies in the non-empty walk voxel with the
        // largest first index P <= q; its slot is q + (start - P).  S.off holds
        // start - P by rank among the non-empty walk voxels.
        W.end = incl;
        W.p1 = incl - wc1;
        W.p0 = W.p1 - wc0;
        W.mark(S, 0);       // cleared before the task
        {
            const unsigned N0 = __ballot_sync(full, wc0 > 0), N1 = __ballot_sync(full, wc1 > 0);
            const int k = __popc(N0 & lt) + __popc(N1 & lt);
            if (wc0 > 0) S.off[k] = st0 - W.p0;
            if (wc1 > 0) S.off[k + (wc0 > 0)] = st1 - W.p1;
        }
        // the homes' own walk indices: the task's voxel is the second one of lane 8
        // (of another one, or of none, in a truncated walk, which no tiled scene has)
        int q_self;
        if (kLayout == 1) {
            const int P = __shfl_sync(full, W.p1, 8), Pb = __shfl_sync(full, W.p0, 9);
            q_self = ih < c_a ? P + (d0 - vst) + ih : Pb + ih - c_a;
        } else {
            const unsigned own0 = __ballot_sync(full, wc0 > 0 && id0 == vid);
            const unsigned own1 = __ballot_sync(full, wc1 > 0 && id1 == vid);
            const int P0 = __shfl_sync(full, W.p0, own0 ? __ffs(own0) - 1 : 0);
            const int P1 = __shfl_sync(full, W.p1, own1 ? __ffs(own1) - 1 : 0);
            q_self = own0 | own1 ? (own1 ? P1 : P0) + (d0 - vst) + ih : -1;
        }
        __syncwarp();
        // the homes' side of the contraction (rows lane / 4 and lane / 4 + 8)
        const TcFrame F{((float)vx + 0.5f) * sc.vs[0], ((float)vy + 0.5f) * sc.vs[1],
                        ((float)vz + (pair ? 1.0f : 0.5f)) * sc.vs[2], sc.u_scale};
        uint32_t A[4] = {0u, 0u, 0u, 0u};
        float C0[4] = {1.0f, 1.0f, 1.0f, 1.0f};      // rows without a home accept nothing
        bool ballots = c_t <= kTcBallot || !(sc.u_h2 <= kTcH2);
        if (!ballots) {
            // lanes i and 16 + i split home i; the mma rows of a lane are lane / 4
            // and lane / 4 + 8
            const float x = (pi.x - F.ox) * F.s, y = (pi.y - F.oy) * F.s, z = (pi.z - F.oz) * F.s;
            const float c = x * x + y * y + z * z;
            const uint4 f = split_halves(-2.0f * x, -2.0f * y, -2.0f * z, 1.0f);
            const float tc = c - sc.u_h2;
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int r = (lane >> 2) + 8 * e;
                const uint32_t fx = __shfl_sync(full, f.x, r), fy = __shfl_sync(full, f.y, r);
                const uint32_t fz = __shfl_sync(full, f.z, r), fw = __shfl_sync(full, f.w, r);
                const float tr = __shfl_sync(full, tc, r);
                if (r < c_t) {
                    A[e] = (lane & 1) ? fy : fx;          // (zh, 1) or (xh, yh)
                    A[2 + e] = (lane & 1) ? fw : fz;      // (zl, 0) or (xl, yl)
                    C0[2 * e] = C0[2 * e + 1] = tr;
                }
            }
            // a home outside its voxel (clamped coordinates)
            ballots = __any_sync(full, ih < c_t && !(c <= kTcHome));
        }
        // through an mma of zeros, into the four consecutive registers that the
        // others read in place (as plain values they were copied for each)
        float Cq[4];
        {
            const uint32_t zero[4] = {0u, 0u, 0u, 0u};
            mma_16x8x16(Cq, zero, 0u, 0u, C0);
        }
        // Long walks: each home's 27-bit mask of the walk voxels within h of it
        // (box distance, the walk's culling test), so that batches in voxels
        // that no home can reach are passed over.
        const bool cull = !sc.walk_trunc && !pair && M > kTcCullMin;
        if (cull) {
            // walk voxel 3 col + z is lane 2 col's first (z 0), second (1) or lane 2 col + 1's first (2)
            const unsigned reach = reach_mask(pi, vx, vy, vz, sc);
            unsigned reach1 = 0u;
#pragma unroll
            for (int col = 0; col < 9; ++col) {
                W.reach0 |= (reach >> (3 * col) & 1u) << (2 * col) |
                            (reach >> (3 * col + 2) & 1u) << (2 * col + 1);
                reach1 |= (reach >> (3 * col + 1) & 1u) << (2 * col);
            }
            if (!upper) S.reach1[ih] = reach1;
            __syncwarp();
        }
        // the row may not hold every neighbour
        const bool uncapped = kUncapped && cap > kListCap;
        const float inv_h2 = sc.inv_h2;
        int cnt = 0;       // home ih: accepted candidates so far (self included)
        int others = 0;    // of those, not the particle itself
        Kahan acc;         // lane i: entries of home i below kSumSplit, lane 16 + i: the rest
        Kahan first;       // uncapped: the first part; acc of lane i then sums every entry
        long long unit = 0;      // uncapped: the home's place in the pool, and its length
        int room = 0;
        // Uncapped: the lists that will not fit their rows get room in the pool, as
        // long as the accepted candidates and those of the walk that are still
        // to come.  More of those than a batch, and the walk is decided twice,
        // once to count (counting) and again, chunk by chunk, to list; not when
        // the pool is full.  Room for the rest of any walk, uncounted, left most
        // particles of scenes of 12 and more per voxel without a list (100,000
        // particles, step: 13 per voxel 426 -> 186 us, 20: 632 -> 271).
        bool counting = false, reserve = kUncapped && uncapped && nbr.over;
        if (kUncapped && reserve && M > kTcChunk + kTcBatch) {
            int left = 0;
            if (lane == 0)
                left = *(volatile unsigned long long*)nbr.over_used < nbr.over_units;
            counting = reserve = __shfl_sync(full, left, 0);
        }
        for (int c0 = 0; c0 < M; c0 += kTcChunk) {
            const int c1 = min(M, c0 + kTcChunk);
            int T, gh, Th;
            const int G = tc_decide(S, T, gh, Th, cnt, c_t, cap, c0, c1, W, cull, A, Cq, ballots, F, pi,
                                    pos, n, sc);
            if (kUncapped && reserve) {
                const int seen = min(cnt + T, cap);
                const bool all = !counting || c1 == M || !__any_sync(full, home && seen < cap);
                if (all) {
                    const int most = counting ? seen : min(cnt + T + M - c1, cap);
                    const int need = home && most > kListCap ? (most + 7) >> 3 : 0;
                    int incl = need;
#pragma unroll
                    for (int o = 1; o < kTaskRun; o <<= 1) {
                        const int v = __shfl_up_sync(full, incl, o);
                        if (lane >= o) incl += v;
                    }
                    const int total = __shfl_sync(full, incl, kTaskRun - 1);
                    unsigned long long u = 0;
                    if (lane == 0 && total) u = atomicAdd(nbr.over_used, (unsigned long long)total);
                    u = __shfl_sync(full, u, 0);
                    if (need && u + total <= nbr.over_units) {
                        unit = (long long)u + incl - need;
                        room = 8 * need;
                    }
                    reserve = false;
                }
                if (counting) {
                    cnt = seen;
                    if (!all) continue;
                    counting = false;
                    cnt = 0;
                    __syncwarp();       // every lane is done with the marks
                    if (lane < kTcWords) S.seg[lane] = 0u;
                    __syncwarp();
                    W.mark(S, 0);
                    __syncwarp();
                    c0 = -kTcChunk;
                    continue;
                }
            }
            const int n_all = ih < c_t ? max(min(T, cap - cnt), 0) : 0;   // entries used here
            int n_lo = min(n_all, max(kSumSplit - cnt, 0)), n_hi = n_all - n_lo;
            // where the lane starts: the lower one at the first word, the upper
            // one after the n_lo entries of the lower one
            const int g0 = upper && n_hi > 0 ? gh : 0;
            uint32_t w0 = S.mask[ih][g0];
            if (g0 | (int)upper) w0 = drop_first(w0, n_hi > 0 ? n_lo - Th : 0);
            TcCursor C(S, ih, g0, w0);
            // the particle itself is accepted and counted, but neither summed
            // nor listed: the upper lane's first list index is one lower when
            // the particle lies before its entries
            const int sq = q_self - c0;
            const uint32_t self = smem_addr(S.cand) + (uint32_t)sq * (uint32_t)sizeof(float4);
            int k = others;
            if (upper) k += n_lo - (sq >= 0 && sq < 32 * g0 + __clz(w0) && sq < 32 * G ? 1 : 0);
            const uint32_t row0 = smem_addr(S.list[ih]);
            const uint32_t row = row0 + 4 * k;
            uint32_t end;
            if (!uncapped) {
                end = tc_sum<false>(C, upper ? n_hi : n_lo, row, 0u, self, pi, inv_h2, acc);
            } else {
                // the lower lane goes over every entry and lists them
                const uint32_t row_end = upper ? row0 : row0 + 4 * kListCap;
                int32_t* over = nbr.over + 8 * unit + others;    // lower lanes
                const uint32_t over_end = row0 + 4 * room;
                end = tc_sum<true>(C, upper ? n_hi : n_lo, row, row_end, self, pi, inv_h2, acc, over,
                                   over_end);
                if (cnt < kSumSplit) first = acc;
                over += (end - row) >> 2;
                end = tc_sum<true>(C, upper ? 0 : n_hi, end, row_end, self, pi, inv_h2, acc, over,
                                   over_end);
            }
            // entries of both lanes (uncapped: the lower lane went over all)
            const int mine = (int)(end - row) >> 2;
            others += uncapped ? __shfl_sync(full, mine, ih)
                               : mine + __shfl_xor_sync(full, mine, 16);
            cnt += T;
            __syncwarp();
            if (!__any_sync(full, home && cnt < cap)) break;
        }
        __syncwarp();
        if (lane < kTcWords) S.seg[lane] = 0u;      // for the next task
        if (kUncapped && home && others > kListCap) {
            S.list[ih][0] = others <= room ? others : 0;
            S.list[ih][1] = (int)unit;
        }
        if (kUncapped) __syncwarp();
        // list rows, four homes at a time, 16 bytes per lane (entries past a
        // row's count are not read by anyone)
        if (nbr.idx) {
#pragma unroll
            for (int i0 = 0; i0 < kTaskRun; i0 += 4) {
                const int i = i0 + (lane >> 3), k = 4 * (lane & 7);
                const int si = __shfl_sync(full, s, i);
                if (i < c_t)
                    *reinterpret_cast<int4*>(nbr.idx + (size_t)si * kListCap + k) =
                        *reinterpret_cast<const int4*>(&S.list[i][k]);
            }
        }
        // lane 16 + i's part joins lane i's; with more neighbours than the row
        // holds the sum is in one part (density_one)
        {
            Kahan rest;
            rest.s = __shfl_down_sync(full, acc.s, 16);
            rest.c = __shfl_down_sync(full, acc.c, 16);
            const bool over = others > kListCap;
            if (uncapped && !over) acc = first;
            if (!over) acc.merge(rest);
            if (home) {
                const float r = (acc.s * sc.w_const) * sc.mass;
                if (rho) rho[s] = r;
                if (kGather) {
                    const float4 v = vel_row(vrows, s, pbegin, n_scenes);
                    vrows.vel_out[s] = v;
                    stg256(fin + 2 * s, force_record_a(pi, sc, r),
                           make_float4(v.x, v.y, v.z, 1.0f / r));
                } else if (fin) {
                    write_force_inputs(s, pi, sc, vel, r, fin);
                }
                if (nbr.count) nbr.count[s] = over ? -1 : others;
            }
        }
        __syncwarp();
    }
}


}  // namespace

cudaError_t launch_density_tc(const Launch& L, const float4* pos, const float4* vel,
                              const int32_t* vstart, const int32_t* vcount, float* rho,
                              float4* fin, NbrList nbr, const int2* tasks,
                              const int32_t* task_count, int32_t* task_next, bool uncapped,
                              const int32_t* task_offset, VelRows vrows) {
    if (L.n == 0) return cudaSuccess;
    // persistent grid: up to 6 blocks of 4 warps per SM (shared memory), warps
    // take tasks in turn; small scenes get about a warp per task, so that the
    // tasks spread over the SMs (a task's latency is most of their pass)
    const int blocks = std::min((L.n + 8 * kTcWarps - 1) / (8 * kTcWarps), device_sm_count() * 6);
    // the velocity gather is for one capped sparse scene (the pipelined host order)
    if (vrows.vel64 && (L.layout != 1 || uncapped)) return cudaErrorInvalidValue;
    auto kernel = vrows.vel64 ? k_density_tc<1, false, true>
                  : uncapped  ? (L.layout == 1   ? k_density_tc<1, true, false>
                                 : L.layout == 2 ? k_density_tc<2, true, false>
                                                 : k_density_tc<0, true, false>)
                              : (L.layout == 1   ? k_density_tc<1, false, false>
                                 : L.layout == 2 ? k_density_tc<2, false, false>
                                                 : k_density_tc<0, false, false>);
    return launch_chained(kernel, blocks, kTcWarps * 32, L, L.scenes, L.pbegin, L.n_scenes,
                          L.n, pos, vel, vstart, vcount, rho, fin, nbr, tasks, task_count,
                          task_next, task_offset, vrows);
}

}  // namespace sphgb
