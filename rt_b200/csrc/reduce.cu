// reduce.cu -- reductions over the wavelengths of a trace's result: the
// transmission per wavelength of the reference's losses_comp
// (efficiency/losses_comp.cpp:11-136) and the distinct wavelengths of
// print_lambda (tools/print_lambda.cpp:12-90), on device arrays.
//
// Both programs sort or scan the wavelengths of every ray on the host.  A
// composite beam has few distinct wavelengths, so here one pass over the rays
// counts them in hash tables (k_distinct) and one block makes the result from
// the distinct values; where there are too many of them, the wavelengths are
// radix-sorted on the device (CUB).  Only the few numbers of the result come
// back.
#include <cub/cub.cuh>

#include <algorithm>

#include "engine.cuh"

namespace rtb {

namespace {

// losses_comp's counting loop (losses_comp.cpp:74-86) over the sorted
// wavelengths: ll[i] = all[i * nl]; ratio[i] = (number of good[k] == ll[i]
// for k in [cp, cp + nl)) / nl, cp advancing by that number.  The window is
// clipped to the good rays (the reference reads past them).  Sequential, as
// the loop is: one thread, a binary search per wavelength.
__global__ void k_loss_windows(const double* all, const double* good, uint64_t n_good, uint64_t n_lambda, uint64_t nl,
                               double* ll, double* ratio) {
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    uint64_t cp = 0;
    for (uint64_t i = 0; i < n_lambda; ++i) {
        const double v = all[i * nl];
        ll[i] = v;
        const uint64_t e = (cp + nl < n_good) ? cp + nl : n_good;
        uint64_t lo = cp, hi = e;  // first index in [cp, e) with good[k] >= v
        while (lo < hi) {
            const uint64_t m = (lo + hi) / 2;
            if (good[m] < v) lo = m + 1; else hi = m;
        }
        uint64_t a = lo, b = e;    // first index in [lo, e) with good[k] > v
        while (a < b) {
            const uint64_t m = (a + b) / 2;
            if (good[m] <= v) a = m + 1; else b = m;
        }
        // equal values are contiguous in sorted order; the reference counts
        // only those inside the window, and they start at lo
        const uint64_t cnt = a - lo;
        ratio[i] = 1.0 * (double)cnt / (double)nl;
        cp += cnt;
        if (cp > n_good) break;
    }
}

// Run heads of sorted wavelengths: the first of each run of equal values
// (NaN equals nothing, as with the reference's ==).
__global__ void k_run_heads(const double* v, uint64_t n, char* head) {
    for (uint64_t k = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; k < n; k += (uint64_t)blockDim.x * gridDim.x)
        head[k] = (k == 0 || !(v[k] == v[k - 1])) ? 1 : 0;
}

__global__ void k_iota(uint64_t n, unsigned long long* idx) {
    for (uint64_t k = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; k < n; k += (uint64_t)blockDim.x * gridDim.x)
        idx[k] = k;
}

size_t al(size_t x) { return (x + 255) / 256 * 256; }

// ---- few distinct wavelengths ----------------------------------------------
// The distinct values of the array with, for each, the number of rays before
// and from n_good on and the first index.  Zeros (two bit patterns, one
// value), NaNs (no value equals them) and more than kMaxDistinct values clear
// *few, and the caller sorts.
constexpr int kMaxDistinct = 1024;
constexpr int kSlots = 2048;        // per block, in shared memory
constexpr int kGlobalSlots = 4096;  // of all blocks
constexpr unsigned long long kNoKey = ~0ull;  // a NaN

struct Distinct {
    unsigned long long* key;    // kGlobalSlots each, all bits set at the start:
    unsigned long long* good;   // no key, and counts from -1 on
    unsigned long long* lost;
    unsigned long long* first;
    unsigned* few;              // all bits set: it is few
    unsigned* used;             // slots taken, from -1 on
};
constexpr size_t kDistinctBytes = 4 * sizeof(unsigned long long) * kGlobalSlots + 256;

Distinct distinct_at(char* p) {
    auto* q = reinterpret_cast<unsigned long long*>(p);
    auto* f = reinterpret_cast<unsigned*>(q + 4 * kGlobalSlots);
    return Distinct{q, q + kGlobalSlots, q + 2 * kGlobalSlots, q + 3 * kGlobalSlots, f, f + 1};
}

__device__ __forceinline__ unsigned slot_hash(unsigned long long k) {
    const unsigned h = ((unsigned)k ^ (unsigned)(k >> 32)) * 0x9E3779B1u;
    return h ^ (h >> 15);
}

// The slot of k in a table, taken if k is not there; -1 when `most` are taken
// (a key too many is not put in: in a full table every further look-up would
// walk all of it, 2000 values of 4e6 rays 50 us).
__device__ __forceinline__ int slot_of(unsigned long long* keys, unsigned mask, unsigned* used, unsigned most,
                                       unsigned long long k) {
    for (unsigned i = slot_hash(k) & mask, tries = 0; tries <= mask; i = (i + 1) & mask, ++tries) {
        unsigned long long at = *(volatile unsigned long long*)(keys + i);
        if (at == kNoKey) {
            if (*(volatile unsigned*)used + 1u >= most) return -1;
            at = atomicCAS(keys + i, kNoKey, k);
            if (at == kNoKey) return atomicAdd(used, 1u) + 1u < most ? (int)i : -1;
        }
        if (at == k) return (int)i;
    }
    return -1;
}

// Bound by the shared-memory look-up and count of each ray (rays in a result
// file's order have their wavelengths in no order): 4e6 rays of 64
// wavelengths in 0.026 ms, 1.2 TB/s; the radix sort it replaces took 0.16 ms
// for keys and 0.33 ms with indices.
constexpr int kDistinctThreads = 512;
__global__ void __launch_bounds__(kDistinctThreads) k_distinct(const double* lambda, uint64_t n, uint64_t n_good,
                                                               uint64_t chunk, Distinct t) {
    __shared__ unsigned long long key[kSlots];
    __shared__ unsigned good[kSlots], lost[kSlots], first[kSlots];
    __shared__ unsigned used;
    for (int j = threadIdx.x; j < kSlots; j += blockDim.x) {
        key[j] = kNoKey;
        good[j] = lost[j] = 0;
        first[j] = ~0u;
    }
    if (threadIdx.x == 0) used = ~0u;
    __syncthreads();
    const uint64_t from = blockIdx.x * chunk, to = (from + chunk < n) ? from + chunk : n;
    constexpr int kAhead = 4;
    bool ok = true;
    for (uint64_t i = from + threadIdx.x; i < to && ok; i += (uint64_t)kAhead * blockDim.x) {
        double v[kAhead];
#pragma unroll
        for (int a = 0; a < kAhead; ++a) {
            const uint64_t at = i + (uint64_t)a * blockDim.x;
            v[a] = (at < to) ? lambda[at] : 1.0;
        }
#pragma unroll
        for (int a = 0; a < kAhead; ++a) {
            const uint64_t at = i + (uint64_t)a * blockDim.x;
            if (at >= to) break;
            const int s = (v[a] < 0.0 || v[a] > 0.0) ? slot_of(key, kSlots - 1, &used, kMaxDistinct,
                                                                (unsigned long long)__double_as_longlong(v[a]))
                                                     : -1;
            if (s < 0) {
                ok = false;
                break;
            }
            atomicAdd((at < n_good ? good : lost) + s, 1u);
            const unsigned rel = (unsigned)(at - from);
            if (rel < *(volatile unsigned*)(first + s)) atomicMin(first + s, rel);
        }
    }
    if (__syncthreads_or(!ok)) {
        if (threadIdx.x == 0) *(volatile unsigned*)t.few = 0u;
        return;
    }
    if (!*(volatile unsigned*)t.few) return;
    for (int j = threadIdx.x; j < kSlots; j += blockDim.x) {
        if (key[j] == kNoKey) continue;
        const int s = slot_of(t.key, kGlobalSlots - 1, t.used, kMaxDistinct, key[j]);
        if (s < 0) {
            *(volatile unsigned*)t.few = 0u;
            return;
        }
        if (good[j]) atomicAdd(t.good + s, (unsigned long long)good[j]);
        if (lost[j]) atomicAdd(t.lost + s, (unsigned long long)lost[j]);
        atomicMin(t.first + s, (unsigned long long)(from + first[j]));
    }
}

// Doubles other than zeros and NaNs in the order of their values.
__device__ __forceinline__ unsigned long long ordered(unsigned long long k) {
    return k ^ ((k >> 63) ? ~0ull : 1ull << 63);
}

constexpr int kFinishThreads = kMaxDistinct;

// The distinct values' slots sorted by value (or by first index) in slot[0,
// count); every thread calls it.  keys: scratch.
__device__ int sorted_slots(const Distinct& t, bool by_first, unsigned long long* keys, int* slot) {
    __shared__ int count;
    if (threadIdx.x == 0) count = 0;
    keys[threadIdx.x] = ~0ull;
    __syncthreads();
    for (int j = threadIdx.x; j < kGlobalSlots; j += kFinishThreads) {
        const unsigned long long k = t.key[j];
        if (k == kNoKey) continue;
        const int p = atomicAdd(&count, 1);
        keys[p] = by_first ? t.first[j] : ordered(k);
        slot[p] = j;
    }
    __syncthreads();
    const int n = count;
    for (int size = 2; size < 2 * n; size *= 2) {  // bitonic, of the next power of two
        for (int stride = size / 2; stride > 0; stride /= 2) {
            const int i = threadIdx.x, k = i ^ stride;
            if (k > i && (keys[i] > keys[k]) == ((i & size) == 0)) {
                const unsigned long long u = keys[i];
                keys[i] = keys[k];
                keys[k] = u;
                const int v = slot[i];
                slot[i] = slot[k];
                slot[k] = v;
            }
            __syncthreads();
        }
    }
    return n;
}

// losses_comp's result from the distinct values: out = [1 (few), ll, ratio].
// Sorted value j holds places [total before j, total up to j) of all the
// sorted wavelengths and [good before j, good up to j) of the good ones, so
// the searches of k_loss_windows are look-ups; its windows stay sequential,
// 1024 of them at a time from shared memory.
__global__ void __launch_bounds__(kFinishThreads) k_loss_finish(Distinct t, uint64_t n_good, uint64_t n_lambda,
                                                                uint64_t nl, double* out) {
    using Scan = cub::BlockScan<unsigned long long, kFinishThreads>;
    __shared__ typename Scan::TempStorage scan;
    __shared__ unsigned long long all[kFinishThreads], good[kFinishThreads], lo[kFinishThreads], hi[kFinishThreads];
    __shared__ int slot[kFinishThreads];
    __shared__ uint64_t cp;
    const int i = threadIdx.x;
    if (i == 0) {
        out[0] = *t.few ? 1.0 : 0.0;
        cp = 0;
    }
    if (!*t.few) return;
    slot[i] = 0;
    const int n = sorted_slots(t, false, all, slot);
    const unsigned long long g = (i < n) ? t.good[slot[i]] + 1 : 0, l = (i < n) ? t.lost[slot[i]] + 1 : 0;
    unsigned long long sum_good, sum_all;
    Scan(scan).InclusiveSum(g, sum_good);
    __syncthreads();
    Scan(scan).InclusiveSum(g + l, sum_all);
    __syncthreads();
    good[i] = sum_good;
    all[i] = sum_all;
    __syncthreads();
    for (uint64_t base = 0; base < n_lambda; base += kFinishThreads) {
        const uint64_t w = base + i;
        if (w < n_lambda) {
            const uint64_t place = w * nl;
            int a = 0, b = n - 1;  // the first value whose places end after `place`
            while (a < b) {
                const int m = (a + b) / 2;
                if (all[m] > place) b = m; else a = m + 1;
            }
            out[1 + w] = __longlong_as_double((long long)t.key[slot[a]]);
            lo[i] = a ? good[a - 1] : 0;
            hi[i] = good[a];
        }
        __syncthreads();
        if (i == 0) {
            uint64_t c = cp;
            const int m = (int)((n_lambda - base < kFinishThreads) ? n_lambda - base : kFinishThreads);
            for (int k = 0; k < m; ++k) {
                const uint64_t e = (c + nl < n_good) ? c + nl : n_good;
                const uint64_t f = min(max((uint64_t)lo[k], c), e), h = min(max((uint64_t)hi[k], f), e);
                out[1 + n_lambda + base + k] = 1.0 * (double)(h - f) / (double)nl;
                c += h - f;
            }
            cp = c;
        }
        __syncthreads();
    }
}

// print_lambda's list from the distinct values: out = [their number + 1 (0: too
// many), the first max_out of them by first occurrence].
__global__ void __launch_bounds__(kFinishThreads) k_unique_finish(Distinct t, int max_out, double* out) {
    __shared__ unsigned long long keys[kFinishThreads];
    __shared__ int slot[kFinishThreads];
    const int i = threadIdx.x;
    if (!*t.few) {
        if (i == 0) out[0] = 0.0;
        return;
    }
    const int n = sorted_slots(t, true, keys, slot);
    if (i == 0) out[0] = (double)n + 1.0;
    if (i < n && i < max_out) out[1 + i] = __longlong_as_double((long long)t.key[slot[i]]);
}

// Counts the distinct values of lambda[0, n) into a table at `mem`.
int count_distinct(const double* lambda, uint64_t n, uint64_t n_good, char* mem, Distinct& t, cudaStream_t s) {
    t = distinct_at(mem);
    RTB_CUDA_TRY(cudaMemsetAsync(mem, 0xff, kDistinctBytes, s));
    const unsigned grid = grid_for(n, kDistinctThreads * 4, 2);
    k_distinct<<<grid, kDistinctThreads, 0, s>>>(lambda, n, n_good, (n + grid - 1) / grid, t);
    RTB_CUDA_TRY(cudaGetLastError());
    return RTB_OK;
}

}  // namespace

}  // namespace rtb

using namespace rtb;

extern "C" int rtb_loss_ratios(const double* lambda, uint64_t n, uint64_t n_good, uint64_t n_lambda, double* ll,
                               double* ratio, void* stream) {
    if (!lambda || !ll || !ratio || n == 0 || n_lambda == 0 || n_good > n) return RTB_BAD_VALUE;
    if (n > (uint64_t)INT32_MAX * 16) return RTB_BAD_VALUE;
    Lock l;
    int st = ensure_init();
    if (st != RTB_OK) return st;
    cudaStream_t s = stream ? (cudaStream_t)stream : engine().stream;
    const uint64_t nl = n / n_lambda;
    // one pass where the wavelengths are few: C1's 64 over 4e6 rays in 0.045 ms
    // on the device against 0.55 ms for the two sorts and the windows' searches
    {
        DevBuf buf;
        if ((st = buf.alloc(kDistinctBytes + (1 + 2 * n_lambda) * sizeof(double), s)) != RTB_OK) return st;
        double* out = reinterpret_cast<double*>(buf.as<char>() + kDistinctBytes);
        Distinct t;
        if ((st = count_distinct(lambda, n, n_good, buf.as<char>(), t, s)) != RTB_OK) return st;
        k_loss_finish<<<1, kFinishThreads, 0, s>>>(t, n_good, n_lambda, nl, out);
        RTB_CUDA_TRY(cudaGetLastError());
        std::vector<double> h(1 + 2 * n_lambda);
        RTB_CUDA_TRY(cudaMemcpyAsync(h.data(), out, h.size() * sizeof(double), cudaMemcpyDeviceToHost, s));
        RTB_CUDA_TRY(cudaStreamSynchronize(s));
        if (h[0] != 0.0) {
            std::copy(h.begin() + 1, h.begin() + 1 + n_lambda, ll);
            std::copy(h.begin() + 1 + n_lambda, h.end(), ratio);
            return RTB_OK;
        }
    }
    size_t t1 = 0, t2 = 0;
    cub::DeviceRadixSort::SortKeys(nullptr, t1, (const double*)nullptr, (double*)nullptr, (int64_t)n, 0, 64, s);
    if (n_good)
        cub::DeviceRadixSort::SortKeys(nullptr, t2, (const double*)nullptr, (double*)nullptr, (int64_t)n_good, 0,
                                       64, s);
    const size_t tmp = t1 > t2 ? t1 : t2;
    const size_t o_good = al(n * 8), o_ll = o_good + al(n_good * 8 + 8), o_r = o_ll + al(n_lambda * 8),
                 o_t = o_r + al(n_lambda * 8);
    DevBuf buf;
    if ((st = buf.alloc(o_t + tmp, s)) != RTB_OK) return st;
    char* p = buf.as<char>();
    double* all = reinterpret_cast<double*>(p);
    double* good = reinterpret_cast<double*>(p + o_good);
    double* d_ll = reinterpret_cast<double*>(p + o_ll);
    double* d_r = reinterpret_cast<double*>(p + o_r);
    void* t = p + o_t;
    size_t tb = tmp;
    RTB_CUDA_TRY(cub::DeviceRadixSort::SortKeys(t, tb, lambda, all, (int64_t)n, 0, 64, s));
    if (n_good) {
        tb = tmp;
        RTB_CUDA_TRY(cub::DeviceRadixSort::SortKeys(t, tb, lambda, good, (int64_t)n_good, 0, 64, s));
    }
    k_loss_windows<<<1, 1, 0, s>>>(all, good, n_good, n_lambda, nl, d_ll, d_r);
    RTB_CUDA_TRY(cudaGetLastError());
    RTB_CUDA_TRY(cudaMemcpyAsync(ll, d_ll, n_lambda * 8, cudaMemcpyDeviceToHost, s));
    RTB_CUDA_TRY(cudaMemcpyAsync(ratio, d_r, n_lambda * 8, cudaMemcpyDeviceToHost, s));
    RTB_CUDA_TRY(cudaStreamSynchronize(s));
    return RTB_OK;
}

extern "C" int rtb_unique_lambdas(const double* lambda, uint64_t n_good, uint64_t max_out, double* out,
                                  uint64_t* n_out, void* stream) {
    if (!n_out || (n_good && !lambda) || (max_out && !out)) return RTB_BAD_VALUE;
    *n_out = 0;
    if (n_good == 0 || max_out == 0) return RTB_OK;
    if (n_good > (uint64_t)INT32_MAX * 16) return RTB_BAD_VALUE;
    Lock l;
    int st = ensure_init();
    if (st != RTB_OK) return st;
    cudaStream_t s = stream ? (cudaStream_t)stream : engine().stream;
    using u64 = unsigned long long;
    const uint64_t n = n_good;
    // as in rtb_loss_ratios: 1.25e6 good rays of C1 in 0.035 ms against 0.40
    {
        const int most = (int)(max_out < (uint64_t)kMaxDistinct ? max_out : (uint64_t)kMaxDistinct);
        DevBuf buf;
        if ((st = buf.alloc(kDistinctBytes + (1 + (size_t)most) * sizeof(double), s)) != RTB_OK) return st;
        double* d_out = reinterpret_cast<double*>(buf.as<char>() + kDistinctBytes);
        Distinct t;
        if ((st = count_distinct(lambda, n, n, buf.as<char>(), t, s)) != RTB_OK) return st;
        k_unique_finish<<<1, kFinishThreads, 0, s>>>(t, most, d_out);
        RTB_CUDA_TRY(cudaGetLastError());
        std::vector<double> h(1 + (size_t)most);
        RTB_CUDA_TRY(cudaMemcpyAsync(h.data(), d_out, h.size() * sizeof(double), cudaMemcpyDeviceToHost, s));
        RTB_CUDA_TRY(cudaStreamSynchronize(s));
        if (h[0] != 0.0) {
            const uint64_t m = std::min<uint64_t>((uint64_t)h[0] - 1, max_out);
            std::copy(h.begin() + 1, h.begin() + 1 + m, out);
            *n_out = m;
            return RTB_OK;
        }
    }
    // (value, first index) of every run of equal values, then by first index
    size_t t1 = 0, t2 = 0, t3 = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, t1, (const double*)nullptr, (double*)nullptr, (const u64*)nullptr,
                                    (u64*)nullptr, (int64_t)n, 0, 64, s);
    cub::DeviceSelect::Flagged(nullptr, t2, (const double*)nullptr, (const char*)nullptr, (double*)nullptr,
                               (u64*)nullptr, (int64_t)n, s);
    cub::DeviceRadixSort::SortPairs(nullptr, t3, (const u64*)nullptr, (u64*)nullptr, (const double*)nullptr,
                                    (double*)nullptr, (int64_t)n, 0, 64, s);
    size_t tmp = t1 > t2 ? t1 : t2;
    tmp = tmp > t3 ? tmp : t3;
    const size_t a8 = al(n * 8);
    const size_t o_idx = 0, o_sv = a8, o_si = 2 * a8, o_head = 3 * a8, o_uv = o_head + al(n), o_ui = o_uv + a8,
                 o_cnt = o_ui + a8, o_fv = o_cnt + 256, o_fi = o_fv + a8, o_t = o_fi + a8;
    DevBuf buf;
    if ((st = buf.alloc(o_t + tmp, s)) != RTB_OK) return st;
    char* p = buf.as<char>();
    u64* idx = reinterpret_cast<u64*>(p + o_idx);
    double* sv = reinterpret_cast<double*>(p + o_sv);
    u64* si = reinterpret_cast<u64*>(p + o_si);
    char* head = p + o_head;
    double* uv = reinterpret_cast<double*>(p + o_uv);
    u64* ui = reinterpret_cast<u64*>(p + o_ui);
    u64* cnt = reinterpret_cast<u64*>(p + o_cnt);
    double* fv = reinterpret_cast<double*>(p + o_fv);
    u64* fi = reinterpret_cast<u64*>(p + o_fi);
    void* t = p + o_t;
    k_iota<<<grid_for(n, 256, 8), 256, 0, s>>>(n, idx);
    size_t tb = tmp;
    // radix sort is stable: within a run the indices stay ascending, the
    // head's is the first occurrence
    RTB_CUDA_TRY(cub::DeviceRadixSort::SortPairs(t, tb, lambda, sv, idx, si, (int64_t)n, 0, 64, s));
    k_run_heads<<<grid_for(n, 256, 8), 256, 0, s>>>(sv, n, head);
    tb = tmp;
    RTB_CUDA_TRY(cub::DeviceSelect::Flagged(t, tb, sv, head, uv, cnt, (int64_t)n, s));
    tb = tmp;
    RTB_CUDA_TRY(cub::DeviceSelect::Flagged(t, tb, si, head, ui, cnt + 1, (int64_t)n, s));
    u64 h_cnt = 0;
    RTB_CUDA_TRY(cudaMemcpyAsync(&h_cnt, cnt, 8, cudaMemcpyDeviceToHost, s));
    RTB_CUDA_TRY(cudaStreamSynchronize(s));
    tb = tmp;
    RTB_CUDA_TRY(cub::DeviceRadixSort::SortPairs(t, tb, ui, fi, uv, fv, (int64_t)h_cnt, 0, 64, s));
    const uint64_t m = h_cnt < max_out ? h_cnt : max_out;
    RTB_CUDA_TRY(cudaMemcpyAsync(out, fv, m * 8, cudaMemcpyDeviceToHost, s));
    RTB_CUDA_TRY(cudaStreamSynchronize(s));
    *n_out = m;
    return RTB_OK;
}
