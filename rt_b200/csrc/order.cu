// order.cu -- the reference's Rearrange on the device.
//
// Beam::Rearrange (common-lib/beam.cpp:574-598) partitions the good prefix
// [0, ng) with two pointers: scanning from the front for lost rays and from
// the back for good rays, it swaps each pair.  The k-th lost ray in [0, N')
// (N' = ng - lost) therefore trades places with the k-th good ray of
// [N', ng) counted from the back; every other ray stays.  Here that pairing
// is computed in parallel from a prefix sum of the lost marks.
//
// reference_order() replays the Rearrange calls of a whole trace from the
// per-ray lost stages (one partition per stage with losses), giving the order
// in which the reference's Beam::Save writes rays: beams of a few hundred rays
// by a warp each, the others all at once in one cooperative launch.
#include <cooperative_groups.h>
#include <cub/cub.cuh>

#include "engine.cuh"
#include "mixed32.cuh"
#include "rowpipe.cuh"

namespace rtb {

namespace {

// Segment s covers positions [start, start + ng) of the order array.
struct Seg {
    uint64_t start, ng;
};

__device__ __forceinline__ int seg_of(const Seg* segs, int n_segs, uint64_t k) {
    int lo = 0, hi = n_segs - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (segs[mid].start <= k) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// Per segment: lost count = rank[start+ng] - rank[start].
__global__ void k_seg_counts(const Seg* segs, int n_segs, const uint32_t* rank, const uint32_t* mark,
                             uint64_t* seg_lost) {
    int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n_segs) return;
    uint64_t a = segs[s].start, b = segs[s].start + segs[s].ng;
    uint64_t ra = rank[a];
    uint64_t rb = (segs[s].ng > 0) ? (uint64_t)rank[b - 1] + mark[b - 1] : ra;
    seg_lost[s] = rb - ra;
}

// Good rays at the back of each segment record their rank from the back.
__global__ void k_back_slots(uint64_t n, const Seg* segs, int n_segs, const uint32_t* mark, const uint32_t* rank,
                             const uint64_t* seg_lost, uint64_t* slot_pos) {
    for (uint64_t k = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; k < n; k += (uint64_t)blockDim.x * gridDim.x) {
        int s = seg_of(segs, n_segs, k);
        uint64_t start = segs[s].start, ng = segs[s].ng, lost = seg_lost[s];
        if (lost == 0 || k >= start + ng) continue;
        uint64_t np = ng - lost;  // N'
        uint64_t j = k - start;
        if (j < np || mark[k]) continue;
        uint64_t lost_before = rank[k] - rank[start];
        uint64_t lost_after = lost - lost_before;                  // mark[k] == 0
        uint64_t good_after = (ng - 1 - j) - lost_after;
        slot_pos[start + good_after] = k;                           // rank from the back
    }
}

// Lost rays at the front swap with their partner.
template <class SwapFn>
__device__ __forceinline__ void pair_front(uint64_t k, const Seg* segs, int n_segs, const uint32_t* mark,
                                           const uint32_t* rank, const uint64_t* seg_lost, const uint64_t* slot_pos,
                                           SwapFn swap) {
    int s = seg_of(segs, n_segs, k);
    uint64_t start = segs[s].start, ng = segs[s].ng, lost = seg_lost[s];
    if (lost == 0 || k >= start + ng || !mark[k]) return;
    uint64_t np = ng - lost;
    if (k - start >= np) return;
    uint64_t r = rank[k] - rank[start];
    swap(k, slot_pos[start + r]);
}

struct Arr7 {
    double* a[7];
};

__global__ void k_swap_arrays(uint64_t n, const Seg* segs, const uint32_t* mark, const uint32_t* rank,
                              const uint64_t* seg_lost, const uint64_t* slot_pos, Arr7 arr, char* flag) {
    for (uint64_t k = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; k < n; k += (uint64_t)blockDim.x * gridDim.x)
        pair_front(k, segs, 1, mark, rank, seg_lost, slot_pos, [&](uint64_t a, uint64_t b) {
            for (int i = 0; i < 7; ++i) {
                double t = arr.a[i][a];
                arr.a[i][a] = arr.a[i][b];
                arr.a[i][b] = t;
            }
            flag[a] = 1;
            flag[b] = 0;
        });
}

__global__ void k_mark_flags(uint64_t ng, const char* flag, uint32_t* mark) {
    for (uint64_t k = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; k < ng; k += (uint64_t)blockDim.x * gridDim.x)
        mark[k] = flag[k] == 0 ? 1u : 0u;
}

// Workspace: mark, rank (uint32) and slot positions (uint64) over n positions.
struct Work {
    DevBuf buf, scan;
    uint32_t *mark, *rank;
    uint64_t *slot, *seg_lost;
    Seg* segs;
    size_t scan_bytes = 0;
    int init(uint64_t n, int n_segs, cudaStream_t st) {
        size_t bytes = n * 8 + n * 8 + 64 + n_segs * (sizeof(Seg) + 8) + 64;
        int s = buf.alloc(bytes, st);
        if (s != RTB_OK) return s;
        char* p = buf.as<char>();
        slot = reinterpret_cast<uint64_t*>(p);
        p += n * 8;
        mark = reinterpret_cast<uint32_t*>(p);
        p += n * 4;
        rank = reinterpret_cast<uint32_t*>(p);
        p += n * 4 + 64;
        segs = reinterpret_cast<Seg*>(p);
        p += n_segs * sizeof(Seg);
        seg_lost = reinterpret_cast<uint64_t*>(p);
        cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, mark, rank, (int64_t)n, st);
        return scan.alloc(scan_bytes, st);
    }
    int exclusive_scan(uint64_t n, cudaStream_t st) {
        RTB_CUDA_TRY(cub::DeviceScan::ExclusiveSum(scan.p, scan_bytes, mark, rank, (int64_t)n, st));
        return RTB_OK;
    }
};

}  // namespace

namespace {

// The replay of a whole trace's Rearrange calls (k_replay).  A segment (beam)
// is cut into tiles of kTile positions; `stage` holds the lost stage of the
// ray at each position, a tile's kTile bytes together, and follows the swaps.
// Beams of up to kSmallSeg rays are replayed by k_replay_small.
constexpr int kTile = 4096, kReplayThreads = 256, kPer = kTile / kReplayThreads;

struct ReplaySeg {
    uint64_t start;          // position of its first ray
    uint32_t n, ng;          // rays, good ones before the stage at hand
    uint32_t lost, pairs;    // of the stage at hand: rays lost, swaps
    uint32_t tile0, pad;     // its first tile
};

struct Replay {
    ReplaySeg* segs;
    int n_segs, n_stages;
    uint32_t n_tiles;
    const uint8_t* lost_stage;
    uint32_t* order;         // beam-local index of the ray at each position
    uint8_t* stage;
    uint32_t* tile_lost;     // rays of a tile lost at the stage at hand
    uint32_t *front, *back;  // the k-th lost ray's position, and its partner's (at segment start + k)
    unsigned* any;           // bit mask of the stages that lost rays
};

__device__ __forceinline__ int seg_of_tile(const Replay& r, uint32_t t) {
    int lo = 0, hi = r.n_segs - 1;
    while (lo < hi) {  // the last segment that starts at or before tile t
        const int mid = (lo + hi + 1) >> 1;
        if (r.segs[mid].tile0 <= t) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// Bit i: of the thread's kPer positions from j0 on, position j0 + i lies
// before `end` and its ray was lost at stage `st`.
__device__ __forceinline__ unsigned lost_bits(const Replay& r, uint32_t t, uint32_t j0, uint32_t end, unsigned st) {
    if (j0 >= end) return 0;
    const uint4 w = *reinterpret_cast<const uint4*>(r.stage + (size_t)t * kTile + threadIdx.x * kPer);
    const unsigned v[4] = {w.x, w.y, w.z, w.w};
    unsigned bits = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const unsigned eq = __vcmpeq4(v[q], st * 0x01010101u) & 0x08040201u;
        bits |= ((eq | eq >> 8 | eq >> 16 | eq >> 24) & 0xfu) << (4 * q);
    }
    const uint32_t left = end - j0;
    return left < kPer ? bits & ((1u << left) - 1u) : bits;
}

// Sum over the block, to every thread.
__device__ __forceinline__ unsigned block_sum(unsigned v, unsigned* s_warp) {
    v = __reduce_add_sync(0xffffffffu, v);
    if ((threadIdx.x & 31) == 0) s_warp[threadIdx.x >> 5] = v;
    __syncthreads();
    unsigned sum = 0;
    for (int w = 0; w < kReplayThreads / 32; ++w) sum += s_warp[w];
    __syncthreads();
    return sum;
}

// Every stage in turn, the whole grid together; a stage that lost no ray is
// passed over.  Per stage: count each tile's lost rays; with the sums before
// its tiles (and so the number of rays that stay, N'), every block lists the
// front's lost rays by rank and the back's good rays by rank from the back;
// swap the pairs, spread over all of the segment's tiles.  Bound by latency:
// three grid barriers a stage and the scattered reads of the swaps.  C1's 31
// beams, 4e6 rays, losses at 5 of 21 stages: 0.18 ms; 1.5 ms as six kernels
// and a library scan over 32-bit marks for each of the 21 stages, mostly the
// gaps between 168 launches.
__global__ void __launch_bounds__(kReplayThreads, 4) k_replay(Replay r) {
    auto grid = cooperative_groups::this_grid();
    __shared__ unsigned s_warp[kReplayThreads / 32];
    using Scan = cub::BlockScan<unsigned, kReplayThreads>;
    __shared__ typename Scan::TempStorage s_scan;
    // a contiguous run of tiles per block: the sums before them are made once
    // per segment and block
    const uint32_t t0 = (uint32_t)((uint64_t)r.n_tiles * blockIdx.x / gridDim.x);
    const uint32_t t1 = (uint32_t)((uint64_t)r.n_tiles * (blockIdx.x + 1) / gridDim.x);
    const int first_seg = t0 < t1 ? seg_of_tile(r, t0) : 0;
    // the segment of the next tile; tiles are visited in order
    auto advance = [&](int s, uint32_t t) {
        while (s + 1 < r.n_segs && r.segs[s + 1].tile0 <= t) ++s;
        return s;
    };
    unsigned seen[3] = {0, 0, 0};
    int s = first_seg;
    for (uint32_t t = t0; t < t1; ++t) {
        s = advance(s, t);
        const uint32_t j0 = (t - r.segs[s].tile0) * kTile, len = min((uint32_t)kTile, r.segs[s].n - j0);
        const uint64_t at = r.segs[s].start + j0;
        uint8_t v[kPer];  // all loads in flight at once
#pragma unroll
        for (int i = 0; i < kPer; ++i) {
            const uint32_t j = threadIdx.x + i * kReplayThreads;
            v[i] = j < len ? r.lost_stage[at + j] : (uint8_t)RTB_NOT_LOST;
        }
#pragma unroll
        for (int i = 0; i < kPer; ++i) {
            const uint32_t j = threadIdx.x + i * kReplayThreads;
            if (j >= len) break;
            r.stage[(size_t)t * kTile + j] = v[i];
            r.order[at + j] = j0 + j;
            if (v[i] < r.n_stages) {
                const unsigned bit = 1u << (v[i] & 31);
                if (v[i] < 32) seen[0] |= bit;
                else if (v[i] < 64) seen[1] |= bit;
                else seen[2] |= bit;
            }
        }
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const unsigned m = __reduce_or_sync(0xffffffffu, seen[q]);
        if (m && (threadIdx.x & 31) == 0) atomicOr(r.any + q, m);
    }
    grid.sync();
    for (int st = 0; st < r.n_stages; ++st) {
        if (!(r.any[st >> 5] >> (st & 31) & 1u)) continue;
        s = first_seg;
        for (uint32_t t = t0; t < t1; ++t) {
            s = advance(s, t);
            const uint32_t j0 = (t - r.segs[s].tile0) * kTile + threadIdx.x * kPer;
            const unsigned c = block_sum(__popc(lost_bits(r, t, j0, r.segs[s].ng, st)), s_warp);
            if (threadIdx.x == 0) r.tile_lost[t] = c;
        }
        grid.sync();
        s = first_seg;
        int sums_of = -1;
        uint32_t before = 0, total = 0;
        for (uint32_t t = t0; t < t1; ++t) {
            s = advance(s, t);
            const ReplaySeg& g = r.segs[s];
            if (sums_of != s) {
                const uint32_t g1 = g.tile0 + (uint32_t)(((uint64_t)g.n + kTile - 1) / kTile);
                unsigned b = 0, a = 0;
                for (uint32_t q = g.tile0 + threadIdx.x; q < g1; q += kReplayThreads) {
                    const unsigned c = r.tile_lost[q];
                    a += c;
                    if (q < t) b += c;
                }
                before = block_sum(b, s_warp);
                total = block_sum(a, s_warp);
                sums_of = s;
            }
            if (t == g.tile0 && threadIdx.x == 0) r.segs[s].lost = total;
            const uint32_t in_tile = r.tile_lost[t], ng = g.ng, keep = ng - total;  // keep: N'
            const uint32_t tile_j = (t - g.tile0) * kTile;
            const bool holds_keep = total && tile_j <= keep && keep - tile_j < kTile;
            // a front tile without lost rays and a back tile without good ones list nothing
            const bool idle =
                total == 0 || tile_j >= ng ||
                (!holds_keep && (tile_j < keep ? in_tile == 0 : in_tile == min((uint32_t)kTile, ng - tile_j)));
            if (!idle) {
                const uint32_t j0 = tile_j + threadIdx.x * kPer;
                const unsigned bits = lost_bits(r, t, j0, ng, st);
                unsigned rank;
                Scan(s_scan).ExclusiveSum(__popc(bits), rank);
                __syncthreads();
                rank += before;  // rays of the segment lost before position j0
                uint32_t* const front = r.front + g.start;
                uint32_t* const back = r.back + g.start;
                const unsigned have = j0 >= ng ? 0u : ng - j0 < kPer ? (1u << (ng - j0)) - 1u : (1u << kPer) - 1u;
                // the positions before N'
                const unsigned fore = j0 >= keep ? 0u : keep - j0 < kPer ? (1u << (keep - j0)) - 1u : (1u << kPer) - 1u;
                for (unsigned m = bits & fore; m; m &= m - 1)
                    front[rank + __popc(bits & ((m & -m) - 1u))] = j0 + __ffs(m) - 1;
                for (unsigned m = have & ~bits & ~fore; m; m &= m - 1) {
                    const uint32_t j = j0 + __ffs(m) - 1;
                    back[(ng - 1 - j) - (total - rank - __popc(bits & ((m & -m) - 1u)))] = j;
                }
                if (j0 <= keep && keep - j0 < kPer) r.segs[s].pairs = rank + __popc(bits & fore);
            } else if (total == 0 && t == g.tile0 && threadIdx.x == 0) {
                r.segs[s].pairs = 0;
            }
            before += in_tile;
        }
        grid.sync();
        s = first_seg;
        for (uint32_t t = t0; t < t1; ++t) {
            s = advance(s, t);
            ReplaySeg& g = r.segs[s];
            // the pairs spread over all of the segment's tiles
            const uint32_t pairs = g.pairs, tiles = (uint32_t)(((uint64_t)g.n + kTile - 1) / kTile);
            for (uint64_t k = (uint64_t)(t - g.tile0) * kReplayThreads + threadIdx.x; k < pairs;
                 k += (uint64_t)tiles * kReplayThreads) {
                const uint32_t a = r.front[g.start + k], b = r.back[g.start + k];
                const uint32_t o = r.order[g.start + a];
                r.order[g.start + a] = r.order[g.start + b];
                r.order[g.start + b] = o;
                // position b leaves the good rays: its stage is not read again
                r.stage[(size_t)g.tile0 * kTile + a] = r.stage[(size_t)g.tile0 * kTile + b];
            }
            if (t == g.tile0 && threadIdx.x == 0) g.ng -= g.lost;
        }
        grid.sync();
    }
}

// A beam of few rays, by one warp: its rays' stages and order in shared memory,
// the stages that lost rays in turn, with the pairing of k_replay (ranks from
// ballots, 32 positions at a time).  A tile of k_replay per beam would cost a
// block three barriers a stage and kTile bytes of `stage` whatever the beam's
// size: 1e5 beams of 10 rays took 11.3 ms and 410 MB so, 2.5 ms and 3 MB this
// way, 1e4 of 100 rays 1.47 and 0.27 ms (the host's check of the beam table
// with it).  The line lies where a tile's bytes come to 8 a ray, so that the
// replay's scratch stays below 16 a ray; 1000 beams of 500 rays take 57 us here,
// of 600 in k_replay 170.
constexpr int kSmallSeg = 512, kSmallWarps = 8;

struct SmallSeg {
    uint64_t start;
    uint32_t n, pad;
};

__global__ void __launch_bounds__(32 * kSmallWarps) k_replay_small(const SmallSeg* segs, int n_segs, int n_stages,
                                                                   const uint8_t* lost_stage, uint32_t* order) {
    __shared__ uint8_t s_stage[kSmallWarps][kSmallSeg];
    __shared__ uint16_t s_order[kSmallWarps][kSmallSeg];
    __shared__ uint16_t s_front[kSmallWarps][kSmallSeg / 2], s_back[kSmallWarps][kSmallSeg / 2];
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5, below = (1u << lane) - 1u;
    uint8_t* const stage = s_stage[warp];
    uint16_t *const ord = s_order[warp], *const front = s_front[warp], *const back = s_back[warp];
    for (int q = (int)(blockIdx.x * kSmallWarps + warp); q < n_segs; q += (int)(gridDim.x * kSmallWarps)) {
        const uint64_t start = segs[q].start;
        const int n = (int)segs[q].n;
        unsigned seen[3] = {0, 0, 0};
        for (int j = (int)lane; j < n; j += 32) {
            const unsigned v = lost_stage[start + j];
            stage[j] = (uint8_t)v;
            ord[j] = (uint16_t)j;
            if (v < (unsigned)n_stages) {
                const unsigned bit = 1u << (v & 31);
                if (v < 32) seen[0] |= bit;
                else if (v < 64) seen[1] |= bit;
                else seen[2] |= bit;
            }
        }
        __syncwarp();
        int ng = n;
#pragma unroll
        for (int w = 0; w < 3; ++w) {
            for (unsigned left = __reduce_or_sync(0xffffffffu, seen[w]); left; left &= left - 1) {
                const unsigned st = 32u * w + __ffs(left) - 1;
                int lost = 0;
                for (int j0 = 0; j0 < ng; j0 += 32) {
                    const int j = j0 + (int)lane;
                    lost += __popc(__ballot_sync(0xffffffffu, j < ng && stage[j] == st));
                }
                const int keep = ng - lost;
                int pairs = 0, backs = 0;
                for (int j0 = 0; j0 < keep; j0 += 32) {  // lost rays at the front
                    const int j = j0 + (int)lane;
                    const bool hit = j < keep && stage[j] == st;
                    const unsigned hits = __ballot_sync(0xffffffffu, hit);
                    if (hit) front[pairs + __popc(hits & below)] = (uint16_t)j;
                    pairs += __popc(hits);
                }
                for (int j0 = ng - 1; j0 >= keep; j0 -= 32) {  // good rays at the back, from the end
                    const int j = j0 - (int)lane;
                    const bool hit = j >= keep && stage[j] != st;
                    const unsigned hits = __ballot_sync(0xffffffffu, hit);
                    if (hit) back[backs + __popc(hits & below)] = (uint16_t)j;
                    backs += __popc(hits);
                }
                __syncwarp();
                for (int k = (int)lane; k < pairs; k += 32) {
                    const int a = front[k], b = back[k];
                    const uint16_t o = ord[a];
                    ord[a] = ord[b];
                    ord[b] = o;
                    stage[a] = stage[b];  // position b leaves the good rays: its stage is not read again
                }
                __syncwarp();
                ng = keep;
            }
        }
        for (int j = (int)lane; j < n; j += 32) order[start + j] = ord[j];
        __syncwarp();
    }
}

// Positions outside every segment, relative to the segment before them (or the
// first); the others are written after this.
__global__ void k_iota(uint64_t n, const uint64_t* starts, int n_segs, uint32_t* order) {
    for (uint64_t k = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; k < n; k += (uint64_t)blockDim.x * gridDim.x) {
        int lo = 0, hi = n_segs - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (starts[mid] <= k) lo = mid; else hi = mid - 1;
        }
        order[k] = (uint32_t)(k - starts[lo]);
    }
}

}  // namespace

int reference_order(const DevBeam* h_beams, int n_beams, int n_stages, const DevRays& rays, uint32_t* order,
                    cudaStream_t st) {
    const uint64_t n = rays.n;
    if (n == 0) return RTB_OK;
    if (n > 0xFFFFFFFFull) return RTB_BAD_VALUE;
    std::vector<ReplaySeg> segs;
    std::vector<SmallSeg> small;
    small.reserve(n_beams);
    uint64_t tiles = 0, covered = 0, end = 0;
    for (int b = 0; b < n_beams; ++b) {
        const uint64_t first = h_beams[b].first_ray;
        const uint32_t nr = (uint32_t)h_beams[b].n_rays;
        if (first < end) return RTB_BAD_VALUE;
        end = first + nr;
        covered += nr;
        if (nr == 0) continue;
        if (nr <= (uint32_t)kSmallSeg) {
            small.push_back(SmallSeg{first, nr, 0});
        } else {
            segs.push_back(ReplaySeg{first, nr, nr, 0, 0, (uint32_t)tiles, 0});
            tiles += (nr + (uint64_t)kTile - 1) / kTile;
        }
    }
    std::vector<uint64_t> starts(covered < n ? n_beams : 0);
    for (size_t b = 0; b < starts.size(); ++b) starts[b] = h_beams[b].first_ray;
    auto al = [](size_t x) { return (x + 255) / 256 * 256; };
    const uint64_t listed = segs.empty() ? 0 : segs.back().start + segs.back().n;
    const size_t o_any = 0, o_segs = 256, o_small = o_segs + al(segs.size() * sizeof(ReplaySeg)),
                 o_starts = o_small + al(small.size() * sizeof(SmallSeg)),
                 o_lost = o_starts + al(starts.size() * sizeof(uint64_t)), o_stage = o_lost + al(tiles * 4),
                 o_front = o_stage + al(tiles * kTile), o_back = o_front + al(listed * 4);
    DevBuf buf;
    int s = buf.alloc(o_back + al(listed * 4), st);
    if (s != RTB_OK) return s;
    char* p = buf.as<char>();
    if (!starts.empty()) {
        uint64_t* d = reinterpret_cast<uint64_t*>(p + o_starts);
        RTB_CUDA_TRY(cudaMemcpyAsync(d, starts.data(), starts.size() * sizeof(uint64_t), cudaMemcpyHostToDevice, st));
        k_iota<<<grid_for(n, 256, 8), 256, 0, st>>>(n, d, (int)starts.size(), order);
    }
    if (!small.empty()) {
        SmallSeg* d = reinterpret_cast<SmallSeg*>(p + o_small);
        RTB_CUDA_TRY(cudaMemcpyAsync(d, small.data(), small.size() * sizeof(SmallSeg), cudaMemcpyHostToDevice, st));
        k_replay_small<<<grid_for(small.size(), kSmallWarps, 8), 32 * kSmallWarps, 0, st>>>(
            d, (int)small.size(), n_stages, rays.lost_stage, order);
    }
    RTB_CUDA_TRY(cudaGetLastError());
    if (segs.empty()) return RTB_OK;
    Replay r;
    r.segs = reinterpret_cast<ReplaySeg*>(p + o_segs);
    r.n_segs = (int)segs.size();
    r.n_stages = n_stages;
    r.n_tiles = (uint32_t)tiles;
    r.lost_stage = rays.lost_stage;
    r.order = order;
    r.stage = reinterpret_cast<uint8_t*>(p + o_stage);
    r.tile_lost = reinterpret_cast<uint32_t*>(p + o_lost);
    r.front = reinterpret_cast<uint32_t*>(p + o_front);
    r.back = reinterpret_cast<uint32_t*>(p + o_back);
    r.any = reinterpret_cast<unsigned*>(p + o_any);
    RTB_CUDA_TRY(cudaMemsetAsync(r.any, 0, 256, st));
    RTB_CUDA_TRY(cudaMemcpyAsync(r.segs, segs.data(), segs.size() * sizeof(ReplaySeg), cudaMemcpyHostToDevice, st));
    int per_sm = 0;
    RTB_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_replay, kReplayThreads, 0));
    // no more blocks than tiles: the barriers cost by the block
    unsigned blocks = grid_for(tiles, 1, per_sm < 4 ? per_sm : 4);
    void* args[] = {&r};
    RTB_CUDA_TRY(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(k_replay), dim3(blocks),
                                             dim3(kReplayThreads), args, 0, st));
    return RTB_OK;
}

// Beam::Rearrange over host arrays: the lost rays are counted first; none, and
// nothing moves.  A swap touches two rays, so where few are lost the kernel
// swaps them in the host arrays themselves when those are library vectors;
// many are swapped in device copies, 57 bytes a ray each way at the link's full
// rate.  In place against copies, us: 1e4 rays of which 1/64 / 1/4 lost 91/148
// and 96/147; 1e5 of which 1/64 / 1/8 / 1/4 133/343, 273/350 and 363/356; 1e6 of
// which 1/128 / 1/64 / 1/32 902/2193, 1553/2221 and 2264/2228.
constexpr size_t kSwapInPlace = 64;       // at most one ray in this many lost,
constexpr size_t kSwapInPlaceRays = 2048;  // or no more than this
int rearrange_host(size_t ng, double* const host[7], char* flag, size_t* ng_out, cudaStream_t st) {
    Work w;
    int s = w.init(ng, 1, st);
    if (s != RTB_OK) return s;
    bool vectors = true;  // the seven arrays: the flags may lie elsewhere (the reference's do)
    char* dflag = flag;
    DevBuf fbuf, buf;
    if (!in_host_vector(flag, ng, 1)) {
        if ((s = fbuf.alloc(ng, st)) != RTB_OK) return s;
        dflag = fbuf.as<char>();
        RTB_CUDA_TRY(cudaMemcpyAsync(dflag, flag, ng, cudaMemcpyHostToDevice, st));
    }
    Seg seg{0, ng};
    RTB_CUDA_TRY(cudaMemcpyAsync(w.segs, &seg, sizeof(Seg), cudaMemcpyHostToDevice, st));
    const unsigned grid = grid_for(ng, 256, 8);
    k_mark_flags<<<grid, 256, 0, st>>>(ng, dflag, w.mark);
    if ((s = w.exclusive_scan(ng, st)) != RTB_OK) return s;
    k_seg_counts<<<1, 32, 0, st>>>(w.segs, 1, w.rank, w.mark, w.seg_lost);
    uint64_t lost = 0;
    RTB_CUDA_TRY(cudaMemcpyAsync(&lost, w.seg_lost, sizeof(lost), cudaMemcpyDeviceToHost, st));
    RTB_CUDA_TRY(cudaStreamSynchronize(st));
    if (lost == 0) {
        *ng_out = ng;
        return RTB_OK;
    }
    Arr7 arr;
    const bool in_place = lost <= ng / kSwapInPlace || lost <= kSwapInPlaceRays;
    for (int i = 0; i < 7; ++i) {
        vectors = vectors && in_host_vector(host[i], ng * sizeof(double), sizeof(double));
        for (int j = 0; j < i; ++j)  // an array given twice is swapped once
            vectors = vectors && (host[i] + ng <= host[j] || host[j] + ng <= host[i]);
    }
    const bool copies = !(vectors && in_place);
    if (copies && (s = buf.alloc(7 * ng * sizeof(double), st)) != RTB_OK) return s;
    // the flags too: many single bytes stored over the link took 0.25 ms of 2.45
    // (1e6 rays, 40 % lost)
    if (copies && dflag == flag) {
        if ((s = fbuf.alloc(ng, st)) != RTB_OK) return s;
        dflag = fbuf.as<char>();
        RTB_CUDA_TRY(cudaMemcpyAsync(dflag, flag, ng, cudaMemcpyHostToDevice, st));
    }
    for (int i = 0; i < 7; ++i) {
        arr.a[i] = copies ? buf.as<double>() + (size_t)i * ng : host[i];
        if (copies) RTB_CUDA_TRY(cudaMemcpyAsync(arr.a[i], host[i], ng * sizeof(double), cudaMemcpyHostToDevice, st));
    }
    k_back_slots<<<grid, 256, 0, st>>>(ng, w.segs, 1, w.mark, w.rank, w.seg_lost, w.slot);
    k_swap_arrays<<<grid, 256, 0, st>>>(ng, w.segs, w.mark, w.rank, w.seg_lost, w.slot, arr, dflag);
    RTB_CUDA_TRY(cudaGetLastError());
    if (copies)
        for (int i = 0; i < 7; ++i)
            RTB_CUDA_TRY(cudaMemcpyAsync(host[i], arr.a[i], ng * sizeof(double), cudaMemcpyDeviceToHost, st));
    if (dflag != flag) RTB_CUDA_TRY(cudaMemcpyAsync(flag, dflag, ng, cudaMemcpyDeviceToHost, st));
    RTB_CUDA_TRY(cudaStreamSynchronize(st));
    *ng_out = ng - lost;  // only now: a call that fails leaves the caller's count with its rays
    return RTB_OK;
}

// ---------------------------------------------------------------------------
// Coherent tracing order of generated rays.  A composite beam interleaves its
// wavelengths (ray j has wavelength j mod n_lambda) and draws positions
// independently, so the 32 rays of a warp go to 32 wavelengths and 32 points
// of the pupil, and which surface loses each of them is close to random: the
// lanes of rays lost early idle while the others finish the scheme.  Sorted
// by (beam, chunk of 2^chunk_shift consecutive rays, wavelength, Morton code
// of the entrance position), a warp traces neighbouring rays of one
// wavelength, which mostly share their fate.  The key only orders the work:
// any key gives a permutation.

__device__ __forceinline__ uint32_t spread12(uint32_t v) {
    v &= 0xfffu;
    v = (v | (v << 8)) & 0x00ff00ffu;
    v = (v | (v << 4)) & 0x0f0f0f0fu;
    v = (v | (v << 2)) & 0x33333333u;
    v = (v | (v << 1)) & 0x55555555u;
    return v;
}

__global__ void k_order_keys(const GenBeam* beams, int n_beams, uint64_t total, DevRays rays,
                             unsigned long long* keys, uint32_t* idx, int chunk_shift) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < total;
         i += (uint64_t)blockDim.x * gridDim.x) {
        int lo = 0, hi = n_beams - 1;
        while (lo < hi) {
            int mid = (lo + hi + 1) >> 1;
            if (beams[mid].first_ray <= i) lo = mid; else hi = mid - 1;
        }
        const GenBeam& b = beams[lo];
        const uint64_t j = i - b.first_ray;
        const uint64_t lam = (j < b.n_rays && b.n_lambda > 0) ? j % b.n_lambda : 0;
        const double R = b.disk[2] > 0 ? b.disk[2] : 1.0;
        auto q = [R](double v, double c) {
            double u = (v - c) / (2.0 * R) + 0.5;
            u = u < 0.0 ? 0.0 : (u > 1.0 ? 1.0 : u);
            return (uint32_t)(u * 4095.0);
        };
        const uint32_t m = spread12(q(rays.X[i], b.center[0])) | (spread12(q(rays.Y[i], b.center[1])) << 1);
        const uint64_t chunk = j >> chunk_shift;
        keys[i] = ((unsigned long long)(lo & 0xffff) << 48) | ((unsigned long long)(chunk & 0xfffu) << 36) |
                  ((unsigned long long)(lam & 0xfffu) << 24) | m;
        idx[i] = (uint32_t)i;
    }
}

int coherent_order(const GenBeam* d_beams, int n_beams, uint64_t n, const DevRays& rays, uint32_t* order,
                   int chunk_shift, cudaStream_t st) {
    if (n == 0) return RTB_OK;
    if (n > 0xffffffffull) return RTB_BAD_VALUE;
    DevBuf buf;
    const size_t kb = (n * 8 + 255) / 256 * 256, ib = (n * 4 + 255) / 256 * 256;
    size_t tmp = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, tmp, (unsigned long long*)nullptr, (unsigned long long*)nullptr,
                                    (uint32_t*)nullptr, (uint32_t*)nullptr, (int64_t)n, 0, 64, st);
    int s = buf.alloc(2 * kb + ib + tmp + 256, st);
    if (s != RTB_OK) return s;
    char* p = buf.as<char>();
    auto* k_in = reinterpret_cast<unsigned long long*>(p);
    auto* k_out = reinterpret_cast<unsigned long long*>(p + kb);
    auto* i_in = reinterpret_cast<uint32_t*>(p + 2 * kb);
    void* t = p + 2 * kb + ib;
    k_order_keys<<<grid_for(n, 256, 8), 256, 0, st>>>(d_beams, n_beams, n, rays, k_in, i_in, chunk_shift);
    RTB_CUDA_TRY(cudaGetLastError());
    RTB_CUDA_TRY(cub::DeviceRadixSort::SortPairs(t, tmp, k_in, k_out, i_in, order, (int64_t)n, 0, 64, st));
    return RTB_OK;
}

__global__ void k_gather_rays(const uint32_t* order, uint64_t n, DevRays src, DevRays dst) {
    for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < n; t += (uint64_t)blockDim.x * gridDim.x) {
        const uint64_t i = order[t];
        dst.X[t] = src.X[i];
        dst.Y[t] = src.Y[i];
        dst.Z[t] = src.Z[i];
        dst.cX[t] = src.cX[i];
        dst.cY[t] = src.cY[i];
        dst.cZ[t] = src.cZ[i];
        dst.lambda[t] = src.lambda[i];
        dst.flag[t] = src.flag[i];
    }
}

// Row blocks of the tracing order (rowpipe.cuh): slot t goes to element
// t % 32 of row t / 32; the slots after the last ray, up to a whole row, get
// flag 0.  Each thread writes one slot, so a warp writes 32 consecutive
// elements of each component.
__global__ void k_gather_rows64(const uint32_t* order, uint64_t n, DevRays src, void* rows) {
    Row64* dst = static_cast<Row64*>(rows);
    const uint64_t total = (n + 31) / 32 * 32;
    for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < total;
         t += (uint64_t)blockDim.x * gridDim.x) {
        Row64& w = dst[t >> 5];
        const int l = (int)(t & 31);
        if (t < n) {
            const uint64_t i = order ? order[t] : t;
            // the cosines normalised as the kernel would on load (mx::normalize)
            mx::Ray r{src.X[i], src.Y[i], src.Z[i], src.cX[i], src.cY[i], src.cZ[i]};
            mx::normalize(r);
            w.X[l] = r.X;
            w.Y[l] = r.Y;
            w.Z[l] = r.Z;
            w.cX[l] = r.cX;
            w.cY[l] = r.cY;
            w.cZ[l] = r.cZ;
            w.lambda[l] = src.lambda[i];
            w.flag[l] = src.flag[i];
        } else {
            w.X[l] = w.Y[l] = w.Z[l] = w.cX[l] = w.cY[l] = w.cZ[l] = w.lambda[l] = 0.0;
            w.flag[l] = 0;
        }
    }
}

// The same with FP32 positions relative to the ray's beam's origin
// (DevBeam::origin) and FP32 cosines; the wavelength stays FP64.  Both
// gathers store the cosines normalised, so the kernels skip that on rows.
__global__ void k_gather_rows32(const uint32_t* order, uint64_t n, DevRays src, const DevBeam* beams, int n_beams,
                                void* rows) {
    Row32* dst = static_cast<Row32*>(rows);
    const uint64_t total = (n + 31) / 32 * 32;
    for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < total;
         t += (uint64_t)blockDim.x * gridDim.x) {
        Row32& w = dst[t >> 5];
        const int l = (int)(t & 31);
        if (t < n) {
            const uint64_t i = order ? order[t] : t;
            const DevBeam& b = beams[beam_of(beams, n_beams, i)];
            // the FP32 cosines normalised as the kernel would on load (m32::normalize)
            m32::Ray r{(float)(src.X[i] - b.origin[0]), (float)(src.Y[i] - b.origin[1]), (float)(src.Z[i] - b.origin[2]),
                       (float)src.cX[i], (float)src.cY[i], (float)src.cZ[i]};
            m32::normalize(r);
            w.X[l] = r.X;
            w.Y[l] = r.Y;
            w.Z[l] = r.Z;
            w.cX[l] = r.cX;
            w.cY[l] = r.cY;
            w.cZ[l] = r.cZ;
            w.lambda[l] = src.lambda[i];
            w.flag[l] = src.flag[i];
        } else {
            w.X[l] = w.Y[l] = w.Z[l] = w.cX[l] = w.cY[l] = w.cZ[l] = 0.0f;
            w.lambda[l] = 0.0;
            w.flag[l] = 0;
        }
    }
}

}  // namespace rtb
