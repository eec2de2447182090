// gx_radix.cu — stable LSD radix sort / radix partition.
//
// Replaces the CUB DeviceRadixSort calls behind gamax::sort::{sort_column_pair,
// sort_column, argsort} (src/cuda/operators/sort/sort.cu:15-215) and the
// partition wrappers that delegate to them (src/cuda/operators/partition/
// partition.cu:11-99).  Semantics kept: stable, sorts on bits
// [begin_bit, end_bit) of the order-preserving key image (signed ints flip
// the sign bit, floats use the sign-magnitude twiddle with -0.0 == +0.0),
// descending order is stable too.
//
// Two plans:
//   * up to SM_ROWS rows: k_radix_small, every digit pass of the sort in the
//     shared memory of one CTA (one launch);
//   * more rows: k_radix_hist_all reads the keys once and counts every digit
//     of every pass, then one kernel per 8-bit digit (k_radix_onesweep) ranks,
//     places and moves a tile's rows, finding where its digit runs go by a
//     decoupled look-back over the earlier tiles' digit counts (Merrill &
//     Garland, "Single-pass Parallel Prefix Scan with Decoupled Look-back",
//     NVIDIA TR 2016; Adinets & Merrill, "Onesweep: A Faster Least
//     Significant Digit Radix Sort for GPUs", 2022).
// The per-tile plan (k_radix_hist, a scan of the [bin][tile] counts,
// k_radix_scatter per digit) needs no waiting between CTAs and no cleared
// state: it serves the allocation-free sort, and a sort whose look-back gave
// up runs through it again.
#include <algorithm>

#include "gx_groupby.h"

namespace gx {
namespace {

constexpr int RS_NT = 512;
constexpr int RS_WARPS = RS_NT / 32;
constexpr int RS_IPT = 8;
constexpr int RS_TILE = RS_NT * RS_IPT;
constexpr int RS_MAXBITS = 8;
constexpr int RS_BINS = 1 << RS_MAXBITS;

template <int KW>
__device__ __forceinline__ uint64_t load_key(const void* p, int64_t i) {
    if (KW == 4) return __ldg(static_cast<const unsigned*>(p) + i);
    return __ldg(static_cast<const unsigned long long*>(p) + i);
}

template <int KW>
__global__ void __launch_bounds__(RS_NT) k_radix_hist(const void* __restrict__ keys, int64_t n, img_params ip,
                                                       int shift, int dbits, int64_t ntiles,
                                                       int64_t* __restrict__ counts) {
    __shared__ unsigned hist[RS_BINS];
    const int bins = 1 << dbits;
    for (int b = threadIdx.x; b < bins; b += RS_NT) hist[b] = 0;
    __syncthreads();
    int64_t base = blockIdx.x * (int64_t)RS_TILE;
#pragma unroll
    for (int k = 0; k < RS_IPT; ++k) {
        int64_t i = base + k * RS_NT + threadIdx.x;
        if (i < n) {
            uint64_t img = key_image<KW>(load_key<KW>(keys, i), ip);
            unsigned d = (unsigned)((img >> shift) & (uint64_t)(bins - 1));
            atomicAdd(&hist[d], 1u);
        }
    }
    __syncthreads();
    for (int b = threadIdx.x; b < bins; b += RS_NT) counts[(int64_t)b * ntiles + blockIdx.x] = hist[b];
}

template <int KW, int VW, bool IOTA>
__global__ void __launch_bounds__(RS_NT) k_radix_scatter(const void* __restrict__ keys_in,
                                                          const void* __restrict__ vals_in, int64_t n,
                                                          img_params ip, int shift, int dbits,
                                                          int64_t ntiles,
                                                          const int64_t* __restrict__ offsets,
                                                          void* __restrict__ keys_out,
                                                          void* __restrict__ vals_out) {
    using kt = typename std::conditional<KW == 4, uint32_t, unsigned long long>::type;
    using vt = typename std::conditional<VW == 4, uint32_t, unsigned long long>::type;
    extern __shared__ __align__(128) unsigned char smem[];
    unsigned* whist = reinterpret_cast<unsigned*>(smem);                    // [WARPS][BINS]
    int64_t* gbase = reinterpret_cast<int64_t*>(smem + RS_WARPS * RS_BINS * 4);  // [BINS]
    unsigned* dbase = reinterpret_cast<unsigned*>(gbase + RS_BINS);          // [BINS + 1]
    kt* skeys = reinterpret_cast<kt*>(dbase + RS_BINS + 4);
    vt* svals = reinterpret_cast<vt*>(skeys + RS_TILE);

    const int bins = 1 << dbits;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < RS_WARPS * RS_BINS; i += RS_NT) whist[i] = 0;
    __syncthreads();

    const int64_t tile_base = blockIdx.x * (int64_t)RS_TILE;
    const int tile_n = (int)min((int64_t)RS_TILE, n - tile_base);
    const unsigned lt_mask = (1u << lane) - 1u;

    kt key[RS_IPT];
    vt val[RS_IPT];
    unsigned dig[RS_IPT];
    unsigned rank[RS_IPT];
#pragma unroll
    for (int k = 0; k < RS_IPT; ++k) {
        int local = warp * 32 * RS_IPT + k * 32 + lane;  // warp-striped: stable order (k, lane)
        int64_t i = tile_base + local;
        bool valid = local < tile_n;
        key[k] = valid ? (kt)load_key<KW>(keys_in, i) : (kt)0;
        if (VW) {
            if (IOTA) val[k] = (vt)i;
            else if (valid) val[k] = VW == 4 ? (vt)__ldg(static_cast<const unsigned*>(vals_in) + i)
                                             : (vt)__ldg(static_cast<const unsigned long long*>(vals_in) + i);
        }
        unsigned d = valid ? (unsigned)((key_image<KW>((uint64_t)key[k], ip) >> shift) & (uint64_t)(bins - 1))
                           : 0xFFFFu;
        dig[k] = d;
        unsigned peers = __match_any_sync(0xffffffffu, d);
        unsigned r = __popc(peers & lt_mask);
        unsigned prior = valid ? whist[warp * RS_BINS + d] : 0;
        rank[k] = prior + r;
        __syncwarp();
        if (valid && r == 0) whist[warp * RS_BINS + d] = prior + __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    // Exclusive prefix over warps per digit, tile-local digit bases, global bases.
    if (threadIdx.x < RS_BINS) {
        unsigned run = 0;
        if (threadIdx.x < bins) {
            for (int w = 0; w < RS_WARPS; ++w) {
                unsigned c = whist[w * RS_BINS + threadIdx.x];
                whist[w * RS_BINS + threadIdx.x] = run;
                run += c;
            }
        }
        dbase[threadIdx.x] = run;  // digit total for now
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        // exclusive scan of RS_BINS digit totals by one warp (8 per lane)
        unsigned v[RS_BINS / 32];
        unsigned s = 0;
#pragma unroll
        for (int j = 0; j < RS_BINS / 32; ++j) {
            v[j] = dbase[lane * (RS_BINS / 32) + j];
            s += v[j];
        }
        unsigned inc = dev_::warp_inclusive_sum(s);
        unsigned run = inc - s;
#pragma unroll
        for (int j = 0; j < RS_BINS / 32; ++j) {
            dbase[lane * (RS_BINS / 32) + j] = run;
            run += v[j];
        }
    }
    __syncthreads();
    if (threadIdx.x < bins)
        gbase[threadIdx.x] = offsets[(int64_t)threadIdx.x * ntiles + blockIdx.x] - (int64_t)dbase[threadIdx.x];
#pragma unroll
    for (int k = 0; k < RS_IPT; ++k) {
        int local = warp * 32 * RS_IPT + k * 32 + lane;
        if (local < tile_n) {
            unsigned pos = dbase[dig[k]] + whist[warp * RS_BINS + dig[k]] + rank[k];
            skeys[pos] = key[k];
            if (VW) svals[pos] = val[k];
        }
    }
    __syncthreads();
    for (int j = threadIdx.x; j < tile_n; j += RS_NT) {
        kt kk = skeys[j];
        unsigned d = (unsigned)((key_image<KW>((uint64_t)kk, ip) >> shift) & (uint64_t)(bins - 1));
        int64_t o = gbase[d] + j;
        static_cast<kt*>(keys_out)[o] = kk;
        if (VW) static_cast<vt*>(vals_out)[o] = svals[j];
    }
}

size_t scatter_smem(int kw, int vw) {
    return (size_t)RS_WARPS * RS_BINS * 4 + RS_BINS * 8 + (RS_BINS + 4) * 4 + (size_t)RS_TILE * (kw + vw);
}

// The scatter needs more than the default 48 KB of dynamic shared memory,
// so each instantiation's limit is raised once per device before its first
// launch.
template <int KW, int VW, bool IOTA>
void prepare_scatter() {
    static per_device_flag attr;
    attr.once([] {
        GX_CUDA(cudaFuncSetAttribute(k_radix_scatter<KW, VW, IOTA>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)scatter_smem(KW, VW)));
    });
}

template <int KW, int VW, bool IOTA>
void launch_scatter(int64_t ntiles, cudaStream_t s, const void* kin, const void* vin, int64_t n,
                    const img_params& ip, int shift, int dbits, const int64_t* off, void* kout,
                    void* vout) {
    size_t smem = scatter_smem(KW, VW);
    prepare_scatter<KW, VW, IOTA>();
    k_radix_scatter<KW, VW, IOTA><<<(unsigned)ntiles, RS_NT, smem, s>>>(kin, vin, n, ip, shift, dbits,
                                                                       ntiles, off, kout, vout);
    GX_LAUNCHED();
}

void scatter_dispatch(int kw, int vw, bool iota, int64_t ntiles, cudaStream_t s, const void* kin,
                      const void* vin, int64_t n, const img_params& ip, int shift, int dbits,
                      const int64_t* off, void* kout, void* vout) {
#define GX_RS_CASE(K, V, I)                                                                   \
    if (kw == K && vw == V && iota == I) {                                                  \
        launch_scatter<K, V, I>(ntiles, s, kin, vin, n, ip, shift, dbits, off, kout, vout); \
        return;                                                                             \
    }
    GX_RS_CASE(4, 0, false)
    GX_RS_CASE(8, 0, false)
    GX_RS_CASE(4, 4, false)
    GX_RS_CASE(4, 8, false)
    GX_RS_CASE(8, 4, false)
    GX_RS_CASE(8, 8, false)
    GX_RS_CASE(4, 8, true)
    GX_RS_CASE(8, 8, true)
#undef GX_RS_CASE
    fail(GX_EUNSUPPORTED, "radix sort: unsupported key/value width combination");
}

template <int KW>
__global__ void k_image_range(const void* __restrict__ keys, int64_t n, img_params ip,
                              unsigned long long* __restrict__ out) {
    uint64_t lo = ~0ull, hi = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        uint64_t img = key_image<KW>(load_key<KW>(keys, i), ip);
        lo = img < lo ? img : lo;
        hi = img > hi ? img : hi;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        uint64_t l2 = __shfl_xor_sync(0xffffffffu, lo, o), h2 = __shfl_xor_sync(0xffffffffu, hi, o);
        lo = l2 < lo ? l2 : lo;
        hi = h2 > hi ? h2 : hi;
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMin(out, (unsigned long long)lo);
        atomicMax(out + 1, (unsigned long long)hi);
    }
}

template <typename S, typename D>
__global__ void k_narrow(D* __restrict__ out, const S* __restrict__ in, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = (D)in[i];
}

// ---------------------------------------------------------------------------
// One-sweep passes.
// ---------------------------------------------------------------------------
// Image of a key in its own register width, as key_image: zero-extended bits,
// a sign flip (signed integers, floats), all bits flipped for negative floats
// and for a descending sort, minus the bias.  The key type decides `FLT` at
// compile time; the rest are two masks.
template <int KW>
using kreg = typename std::conditional<KW == 8, unsigned long long, uint32_t>::type;

template <int KW, bool FLT>
struct digit_of {
    kreg<KW> flip, bias;
    int shift;
    unsigned mask;
    __device__ __forceinline__ kreg<KW> image(kreg<KW> b) const {
        if constexpr (FLT) {
            constexpr int TOP = 8 * KW - 1;
            if (b == (kreg<KW>(1) << TOP)) b = 0;  // -0.0 sorts as +0.0
            b ^= (b >> TOP) ? ~(kreg<KW>(1) << TOP) : kreg<KW>(0);
        }
        return (b ^ flip) - bias;
    }
    __device__ __forceinline__ unsigned operator()(kreg<KW> b) const { return (unsigned)(image(b) >> shift) & mask; }
};

// The masks of an image: a negative float is all bits flipped, i.e. the sign
// flip of `flip` on top of the other bits flipped in image().
template <int KW, bool FLT>
digit_of<KW, FLT> make_digit(const img_params& ip, int shift, int dbits) {
    digit_of<KW, FLT> d;
    d.flip = ip.kind == VK_U ? kreg<KW>(0) : kreg<KW>(1) << (8 * KW - 1);
    if (ip.desc) d.flip = ~d.flip;
    d.bias = (kreg<KW>)ip.bias;
    d.shift = shift;
    d.mask = (1u << dbits) - 1u;
    return d;
}

template <int KW>
__device__ __forceinline__ kreg<KW> ld_key(const void* p, int64_t i) {
    if constexpr (KW == 1) return __ldg(static_cast<const unsigned char*>(p) + i);
    else if constexpr (KW == 2) return __ldg(static_cast<const unsigned short*>(p) + i);
    else if constexpr (KW == 4) return __ldg(static_cast<const unsigned*>(p) + i);
    else return __ldg(static_cast<const unsigned long long*>(p) + i);
}
template <int KW>
__device__ __forceinline__ void st_key(void* p, int64_t i, kreg<KW> v) {
    if constexpr (KW == 1) static_cast<unsigned char*>(p)[i] = (unsigned char)v;
    else if constexpr (KW == 2) static_cast<unsigned short*>(p)[i] = (unsigned short)v;
    else if constexpr (KW == 4) static_cast<unsigned*>(p)[i] = v;
    else static_cast<unsigned long long*>(p)[i] = v;
}

constexpr int OS_MAX_PASSES = 8;
// What the passes of one sort share: digit counts and, written by the last
// CTA of the histogram kernel, where each digit's rows start and which passes
// run.  A pass whose digit is the same in every row moves nothing and is
// skipped; the others alternate between the two buffers so that the last one
// writes the output.
struct os_plan {
    unsigned long long hist[OS_MAX_PASSES][RS_BINS];
    unsigned long long base[OS_MAX_PASSES][RS_BINS];
    int order[OS_MAX_PASSES];  // position among the passes that run, -1: skipped, or one before it gave up
    int runs;                  // passes that run
    unsigned ticket[OS_MAX_PASSES];
    unsigned done;
    int err;
};

// Digit counts of every pass from one read of the keys: two 1024-thread CTAs
// per SM, 16-byte loads (four in flight per thread) where the column is
// 16-byte aligned, shared histograms.  A digit that all keys of a warp's
// vectors share (constant upper bytes, sorted keys) is counted with one addition.
// 2^28 random int32 keys, four digits: a sort takes 8.58 ms with it, 9.06 when
// every digit of every key was compared across the warp.
constexpr int OH_NT = 1024;
template <int KW, bool FLT>
__global__ void __launch_bounds__(OH_NT, 2) k_radix_hist_all(const void* __restrict__ keys, int64_t n,
                                                             digit_of<KW, FLT> dg, int begin_bit, int end_bit,
                                                             int passes, os_plan* __restrict__ plan) {
    __shared__ unsigned hist[OS_MAX_PASSES][RS_BINS];
    __shared__ int64_t scan_sm[OH_NT / 32 + 1];
    __shared__ int s_last, s_runs;
    for (int i = threadIdx.x; i < OS_MAX_PASSES * RS_BINS; i += OH_NT) (&hist[0][0])[i] = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    auto digit = [&](kreg<KW> img, int p) -> unsigned {
        const int sh = begin_bit + p * RS_MAXBITS;
        const int bits = min(RS_MAXBITS, end_bit - sh);
        return (unsigned)(img >> sh) & ((1u << bits) - 1u);
    };
    // A vector of keys per lane, whole warps: `vary` has the image bits that
    // differ anywhere among them, so digits that do not are counted at once.
    auto add_warp = [&](const kreg<KW>* img, int m) {
        kreg<KW> x = img[0] ^ __shfl_sync(0xffffffffu, img[0], 0);
#pragma unroll
        for (int e = 1; e < 16 / KW; ++e) x |= img[0] ^ img[e];
        kreg<KW> vary;
        if constexpr (KW == 8)
            vary = (unsigned long long)__reduce_or_sync(0xffffffffu, (unsigned)(x >> 32)) << 32 |
                   __reduce_or_sync(0xffffffffu, (unsigned)x);
        else vary = __reduce_or_sync(0xffffffffu, x);
        for (int p = 0; p < passes; ++p) {
            if (digit(vary, p) == 0) {
                if (lane == 0) atomicAdd(&hist[p][digit(img[0], p)], 32u * (unsigned)m);
            } else {
#pragma unroll
                for (int e = 0; e < 16 / KW; ++e) atomicAdd(&hist[p][digit(img[e], p)], 1u);
            }
        }
    };
    auto add_one = [&](kreg<KW> key) {
        const kreg<KW> img = dg.image(key);
        for (int p = 0; p < passes; ++p) atomicAdd(&hist[p][digit(img, p)], 1u);
    };
    const int64_t warps = (int64_t)gridDim.x * (OH_NT / 32);
    const int64_t gw = blockIdx.x * (int64_t)(OH_NT / 32) + (threadIdx.x >> 5);
    constexpr int KPV = 16 / KW, B = KW >= 4 ? 4 : 1;  // keys per vector, vectors per thread and round
    int64_t done = 0;  // rows [0, done) are taken by whole-warp vector rounds
    if ((reinterpret_cast<uintptr_t>(keys) & 15) == 0) {
        const int64_t per = (int64_t)32 * B * KPV, rounds = n / per;
        done = rounds * per;
        const uint4* kv = static_cast<const uint4*>(keys);
        for (int64_t r = gw; r < rounds; r += warps) {
            uint4 x[B];
#pragma unroll
            for (int q = 0; q < B; ++q) x[q] = __ldg(kv + (r * B + q) * 32 + lane);
#pragma unroll
            for (int q = 0; q < B; ++q) {
                const unsigned w[4] = {x[q].x, x[q].y, x[q].z, x[q].w};
                kreg<KW> img[KPV];
#pragma unroll
                for (int e = 0; e < KPV; ++e) {
                    if constexpr (KW == 8) img[e] = dg.image(((unsigned long long)w[2 * e + 1] << 32) | w[2 * e]);
                    else if constexpr (KW == 4) img[e] = dg.image(w[e]);
                    else img[e] = dg.image((w[e * KW / 4] >> (8 * (e * KW % 4))) & ((1u << (8 * KW)) - 1u));
                }
                add_warp(img, KPV);
            }
        }
    }
    for (int64_t i = done + blockIdx.x * (int64_t)OH_NT + threadIdx.x; i < n; i += (int64_t)gridDim.x * OH_NT)
        add_one(ld_key<KW>(keys, i));
    __syncthreads();
    for (int i = threadIdx.x; i < passes * RS_BINS; i += OH_NT) {
        const unsigned c = (&hist[0][0])[i];
        if (c) atomicAdd(&plan->hist[0][0] + i, (unsigned long long)c);
    }
    // The last CTA to finish scans the counts and chooses the passes.
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        s_last = atomicAdd(&plan->done, 1u) == gridDim.x - 1;
        s_runs = 0;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (int p = 0; p < passes; ++p) {
        const int64_t c = threadIdx.x < RS_BINS ? (int64_t)__ldcg(&plan->hist[p][threadIdx.x]) : 0;
        int64_t total;
        const int64_t ex = dev_::block_exclusive_sum<OH_NT, int64_t>(c, scan_sm, &total);
        if (threadIdx.x < RS_BINS) plan->base[p][threadIdx.x] = (unsigned long long)ex;
        const int same = __syncthreads_or(c == n);
        if (threadIdx.x == 0) {
            // With no other pass to run, the last one copies the rows.
            const bool run = !same || (p == passes - 1 && s_runs == 0);
            plan->order[p] = run ? s_runs++ : -1;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) plan->runs = s_runs;
}

// Rank of this row among the warp's rows of the same digit, rows in (call,
// lane) order: the lanes of a digit find each other through a shared bit mask
// (one atomicOr and one read), the highest of them adds their number to the
// warp's count and clears the mask.  `wm` must be zero before the first call.
// (The steps of the atomic-OR ranking in NVIDIA's open-source CUB radix sort.)
// On B200 this costs 0.31 ms per 2^28 rows and digit where __match_any_sync
// costs 1.8 ms and eight ballots 0.73 ms (16 warps per CTA, random digits).
__device__ __forceinline__ unsigned warp_rank(unsigned* wm, unsigned* wh, unsigned d, bool valid, int lane) {
    if (valid) atomicOr(&wm[d], 1u << lane);
    __syncwarp();
    const unsigned peers = valid ? wm[d] : 1u << lane;
    const int leader = 31 - __clz(peers);
    const bool lead = valid && lane == leader;
    unsigned prior = 0;
    if (lead) prior = atomicAdd(&wh[d], (unsigned)__popc(peers));
    prior = __shfl_sync(0xffffffffu, prior, leader);  // every lane has read its mask
    if (lead) wm[d] = 0;
    __syncwarp();
    return prior + __popc(peers & ((1u << lane) - 1u));
}

// Digit counts of a tile as its successors see them: one word per (tile,
// digit), flag and value together, so relaxed accesses suffice.  FAIL: a wait
// gave up in this tile or before it; whoever meets it passes it on.
using os_state = unsigned long long;
constexpr os_state OS_AGG = 1ull << 62, OS_INC = 2ull << 62, OS_FAIL = 3ull << 62, OS_VAL = (1ull << 62) - 1;
constexpr int OS_SPIN_LIMIT = 1 << 20;
constexpr uint32_t OS_COPY_WAIT = 1u << 22;
__device__ __forceinline__ os_state ld_state(const os_state* p) {
    os_state v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_state(os_state* p, os_state v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

struct os_args {
    const void *kin, *vin;
    void *ktmp, *vtmp, *kout, *vout;
    int64_t n;
    int pass, iota;
    int spin_limit;      // empty polls before a look-back gives up (0: at once)
    uint32_t copy_limit; // polls of a copy
    os_state* state[2];  // [tile][digit]; the running pass uses one and clears the other
    os_plan* plan;
};

constexpr int OS_NT = 512;
constexpr int OS_WARPS = OS_NT / 32;
constexpr int OS_WIN = 8;  // earlier tiles a look-back reads together

template <int KW, int VW>
__host__ __device__ constexpr int os_smem(int ipt) {
    const int rows = OS_NT * ipt, order = rows * 4, hists = 2 * OS_WARPS * RS_BINS * 4;
    return rows * (KW + VW) + (order > hists ? order : hists);
}
// Rows per thread: as many (at most 16) as let two CTAs share an SM.
template <int KW, int VW>
constexpr int os_ipt_max() {
    int i = 16;
    while (os_smem<KW, VW>(i) > 106 * 1024) --i;
    return i;
}

// One digit pass.  A CTA takes the next tile of OS_NT * IPT rows (atomic
// ticket: every tile it waits on belongs to a CTA that started earlier).  The
// copy engine brings the tile's keys and values into shared memory in their
// order; the warps rank their rows by digit (warp_rank); the CTA publishes its
// digit counts, lists its rows by digit (`order`: digit << 16 | row) and looks
// back for the start of its digit runs; then output position j fetches its
// row's key and value from shared memory and writes them, run by run.
// Bound by shared-memory wavefronts (about 40 per 32 rows: the rank, the list
// and the gathers are random accesses; L1 70% busy, HBM 38%).  2^28 random
// rows per pass, measured over a whole sort: 1.95 ms for int32 keys with int64
// values (3.5 ms with the stable ranking by __match_any_sync, plus 0.9 ms of
// counting per pass), 1.6 ms for int32 with int32, 2.45 ms for int64 with int64.
// Two CTAs of 512 threads with 6144 rows beat three of 4608 rows (9.05 against
// 10.6 ms a sort), one of 1024 threads (9.6 ms) and 768 threads (10.6 ms); a
// look-back window of 8 tiles beats 4 and 16 by 3% and 10%.
// A tile whose look-back gives up, or whose rows did not arrive, writes nothing,
// sets plan->err and takes the later passes off the plan; without its keys it
// also publishes no count, so no other tile places its rows by one.  So none of them ranks the holes of this pass
// against digit starts that were counted from all rows, and every position
// written lies inside its digit's range.  (Reading plan->err at the start of
// each tile instead cost 1.6% of a sort.)
template <int KW, int VW, bool FLT, int IPT>
__global__ void __launch_bounds__(OS_NT, 2) k_radix_onesweep(digit_of<KW, FLT> dg, os_args a) {
    using vt = typename std::conditional<VW == 8, unsigned long long, uint32_t>::type;
    constexpr int TILE = OS_NT * IPT;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) unsigned long long bars[2];
    __shared__ int64_t gbase[RS_BINS];
    __shared__ unsigned wsum[RS_BINS / 32];
    __shared__ unsigned s_tile;
    const int ord = a.plan->order[a.pass];
    if (ord < 0) return;
    const int left = a.plan->runs - 1 - ord;  // passes still to come
    const void* kin = ord == 0 ? a.kin : (left & 1) ? a.kout : a.ktmp;
    const void* vin = ord == 0 ? a.vin : (left & 1) ? a.vout : a.vtmp;
    void* kout = (left & 1) ? a.ktmp : a.kout;
    void* vout = (left & 1) ? a.vtmp : a.vout;
    const bool iota = a.iota && ord == 0;
    // Selected, not indexed: an index would put the arguments on the stack.
    os_state* state = ord & 1 ? a.state[1] : a.state[0];
    os_state* next_state = ord & 1 ? a.state[0] : a.state[1];

    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    unsigned char* skeys = smem;
    vt* svals = reinterpret_cast<vt*>(smem + TILE * KW);
    unsigned* order = reinterpret_cast<unsigned*>(smem + TILE * (KW + VW));
    unsigned* counts = order;  // [warp][digit], before `order`; then the lane masks
    unsigned* wh = counts + warp * RS_BINS;
    unsigned* wm = wh + OS_WARPS * RS_BINS;
    const uint32_t bar0 = dev_::smem_addr(&bars[0]), bar1 = bar0 + 8;
    const bool load_vals = VW > 0 && !iota;
    // Copies start on 16-byte boundaries (tiles are multiples of 16 bytes).
    const bool kbulk = (reinterpret_cast<uintptr_t>(kin) & 15) == 0, vbulk = (reinterpret_cast<uintptr_t>(vin) & 15) == 0;
    if (t == 0) {
        const unsigned tk = atomicAdd(&a.plan->ticket[a.pass], 1u);
        s_tile = tk;
        dev_::mbar_init(bar0, 1);
        dev_::mbar_init(bar1, 1);
        dev_::mbar_init_fence();
        const int64_t base = (int64_t)tk * TILE;
        if (base + TILE <= a.n) {
            if (kbulk) {
                dev_::mbar_arrive_expect_tx(bar0, TILE * KW);
                dev_::bulk_load_g2s(dev_::smem_addr(skeys), static_cast<const unsigned char*>(kin) + base * KW, TILE * KW, bar0);
            }
            if (load_vals && vbulk) {
                dev_::mbar_arrive_expect_tx(bar1, TILE * VW);
                dev_::bulk_load_g2s(dev_::smem_addr(svals), static_cast<const unsigned char*>(vin) + base * VW, TILE * VW, bar1);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < RS_BINS / 128; ++i) {
        reinterpret_cast<uint4*>(wh)[i * 32 + lane] = make_uint4(0, 0, 0, 0);
        reinterpret_cast<uint4*>(wm)[i * 32 + lane] = make_uint4(0, 0, 0, 0);
    }
    __syncthreads();
    const int64_t tile = s_tile;
    const int64_t tile_base = tile * TILE;
    const int tile_n = (int)min((int64_t)TILE, a.n - tile_base);
    const bool full = tile_n == TILE;
    if (t < RS_BINS) st_state(next_state + tile * RS_BINS + t, 0ull);
    auto row_key = [&](int i) -> kreg<KW> {
        if constexpr (KW == 1) return skeys[i];
        else if constexpr (KW == 2) return reinterpret_cast<const unsigned short*>(skeys)[i];
        else if constexpr (KW == 4) return reinterpret_cast<const unsigned*>(skeys)[i];
        else return reinterpret_cast<const unsigned long long*>(skeys)[i];
    };
    int failed = 0;
    if (!(full && kbulk)) {
        for (int i = t; i < tile_n; i += OS_NT) st_key<KW>(skeys, i, ld_key<KW>(kin, tile_base + i));
        __syncthreads();
    } else if (!dev_::mbar_wait_bounded(bar0, 0, a.copy_limit)) {
        failed = 1;
    }
    if constexpr (VW > 0) {
        if (load_vals && !(full && vbulk))  // read after later barriers
            for (int i = t; i < tile_n; i += OS_NT) svals[i] = __ldg(static_cast<const vt*>(vin) + tile_base + i);
    }

    const int local0 = warp * 32 * IPT + lane;  // row (k, lane) of the warp: local0 + 32 k
    unsigned rk[IPT];  // digit << 16 | rank in the warp's rows of the digit
    // Lanes with one digit queue on its word, so a warp whose first rows share a
    // digit (ordered input, constant digits) looks for such rows and ranks them
    // by lane.  2^25 int64 keys with int32 values into 16 parts, runs of 64 equal
    // keys: 312 us a call, 395 without; 2^28 random int32 keys with int64 values:
    // 8.22 ms, 8.20 without.
    auto one_digit = [](unsigned d) { return (bool)__all_sync(0xffffffffu, d == __shfl_sync(0xffffffffu, d, 0)); };
    if (full && one_digit(dg(row_key(local0)))) {
#pragma unroll
        for (int k = 0; k < IPT; ++k) {
            const unsigned d = dg(row_key(local0 + 32 * k));
            if (one_digit(d)) {
                const unsigned prior = wh[d];
                __syncwarp();
                if (lane == 0) wh[d] = prior + 32;
                __syncwarp();
                rk[k] = (prior + lane) | d << 16;
            } else {
                rk[k] = warp_rank(wm, wh, d, true, lane) | d << 16;
            }
        }
    } else if (full) {
#pragma unroll
        for (int k = 0; k < IPT; ++k) {
            const unsigned d = dg(row_key(local0 + 32 * k));
            rk[k] = warp_rank(wm, wh, d, true, lane) | d << 16;
        }
    } else {
#pragma unroll
        for (int k = 0; k < IPT; ++k) {
            const bool valid = local0 + 32 * k < tile_n;
            const unsigned d = valid ? dg(row_key(local0 + 32 * k)) : 0u;
            rk[k] = warp_rank(wm, wh, d, valid, lane) | d << 16;
        }
    }
    auto give_up = [&] {  // thread 0
        atomicExch(&a.plan->err, 1);
        for (int p = a.pass + 1; p < OS_MAX_PASSES; ++p) a.plan->order[p] = -1;
        // Leave no copy in flight into this CTA's shared memory.
        if (full && kbulk) dev_::mbar_wait_bounded(bar0, 0, OS_COPY_WAIT);
        if (full && load_vals && vbulk) dev_::mbar_wait_bounded(bar1, 0, OS_COPY_WAIT);
    };
    if (__syncthreads_or(failed)) {  // the keys did not arrive
        if (t < RS_BINS) st_state(state + tile * RS_BINS + t, OS_FAIL);
        if (t == 0) give_up();
        return;
    }

    // Tile counts per digit; their prefix over the warps and over the digits.
    unsigned tot = 0, incl = 0;
    unsigned* whd = counts + t;
    if (t < RS_BINS) {
#pragma unroll
        for (int w = 0; w < OS_WARPS; ++w) tot += whd[w * RS_BINS];
        st_state(state + tile * RS_BINS + t, (tile == 0 ? OS_INC : OS_AGG) | tot);
        incl = dev_::warp_inclusive_sum(tot);
        if (lane == 31) wsum[warp] = incl;
    }
    __syncthreads();
    unsigned ex = 0;
    if (t < RS_BINS) {
        ex = incl - tot;
        for (int w = 0; w < warp; ++w) ex += wsum[w];
        unsigned run = ex;
#pragma unroll
        for (int w = 0; w < OS_WARPS; ++w) {
            const unsigned c = whd[w * RS_BINS];
            whd[w * RS_BINS] = run;
            run += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < IPT; ++k) rk[k] += wh[rk[k] >> 16];
    __syncthreads();  // the counts' shared memory becomes `order`
#pragma unroll
    for (int k = 0; k < IPT; ++k)
        if (full || local0 + 32 * k < tile_n)
            order[rk[k] & 0xFFFFu] = (rk[k] & ~0xFFFFu) | (unsigned)(local0 + 32 * k);

    // Look back: rows of this digit in the tiles before this one.
    if (t < RS_BINS) {
        os_state before = 0;
        int64_t j = tile - 1;
        if (j >= 0 && a.spin_limit == 0) failed = 1;
        for (int spins = 0; j >= 0 && !failed;) {
            os_state st[OS_WIN];
#pragma unroll
            for (int q = 0; q < OS_WIN; ++q) st[q] = j - q >= 0 ? ld_state(state + (j - q) * RS_BINS + t) : OS_INC;
            int seen = 0;  // predecessors taken of this window
            bool open = true, inc = false;
#pragma unroll
            for (int q = 0; q < OS_WIN; ++q) {
                const os_state f = st[q] & ~OS_VAL;
                if (open && f == OS_FAIL) failed = 1;
                open = open && f != 0 && f != OS_FAIL;
                if (open) {
                    before += st[q] & OS_VAL;
                    ++seen;
                    inc = f == OS_INC;
                    open = !inc;
                }
            }
            if (inc || failed) break;
            j -= seen;
            if (seen == 0) {
                if (++spins > a.spin_limit) { failed = 1; break; }
                __nanosleep(20);
            }
        }
        if (tile > 0) st_state(state + tile * RS_BINS + t, failed ? OS_FAIL : OS_INC | (before + tot));
        gbase[t] = (int64_t)(a.plan->base[a.pass][t] + before) - (int64_t)ex;
    }
    if (load_vals && full && vbulk && !dev_::mbar_wait_bounded(bar1, 0, a.copy_limit)) failed = 1;
    if (__syncthreads_or(failed)) {
        if (t == 0) give_up();
        return;
    }
#pragma unroll
    for (int m = 0; m < IPT; ++m) {
        const int j = t + m * OS_NT;
        if (full || j < tile_n) {
            const unsigned e = order[j];
            const int r = (int)(e & 0xFFFFu);
            const int64_t o = gbase[e >> 16] + j;
            st_key<KW>(kout, o, row_key(r));
            if constexpr (VW > 0) static_cast<vt*>(vout)[o] = iota ? (vt)(tile_base + r) : svals[r];
        }
    }
}

// Every pass of a sort of at most SM_ROWS rows in one CTA: keys and 16-bit row
// positions move through shared memory, the values are fetched once at the
// end.  Bound by the latency of its barriers: 1000 rows of int32 keys in 37 us a
// call, 8192 in 56 us, against 133 and 154 us through histogram, scan and
// scatter launches per digit.
constexpr int SM_NT = 1024, SM_WARPS = SM_NT / 32, SM_IPT = 8;
constexpr int64_t SM_ROWS = SM_NT * SM_IPT;
template <int KW>
constexpr int small_smem() {
    const int rows = (int)SM_ROWS * ((KW == 8 ? 8 : 4) + 2), hists = 2 * SM_WARPS * RS_BINS * 4;
    return rows > hists ? rows : hists;
}

// Up to SR_ROWS rows (the ordering of a small result): every row's place is the
// number of rows before it, counted by all threads of one CTA at once.  A
// group-by of 5,003 rows ordered by its 61 keys: 147 us, 162 through
// k_radix_small (four passes of barriers, 14 us).
constexpr int SR_NT = 1024, SR_ROWS = 256;
template <int KW, bool FLT>
__global__ void __launch_bounds__(SR_NT) k_radix_rank(const void* __restrict__ kin, const void* __restrict__ vin,
                                                      void* __restrict__ kout, void* __restrict__ vout, int n,
                                                      digit_of<KW, FLT> dg, int bits, int vw, int iota) {
    __shared__ kreg<KW> s_img[SR_ROWS];
    __shared__ unsigned s_place[SR_ROWS];
    const int t = threadIdx.x;
    if (t < n) {
        const kreg<KW> img = dg.image(ld_key<KW>(kin, t)) >> dg.shift;
        s_img[t] = bits >= 8 * (int)sizeof(kreg<KW>) ? img : img & ((kreg<KW>(1) << bits) - 1);
        s_place[t] = 0;
    }
    __syncthreads();
    const int i = t & (SR_ROWS - 1);
    constexpr int PARTS = SR_NT / SR_ROWS;
    if (i < n) {
        const int per = (n + PARTS - 1) / PARTS, j0 = (t / SR_ROWS) * per, j1 = min(n, j0 + per);
        const kreg<KW> mine = s_img[i];
        unsigned before = 0;
        for (int j = j0; j < j1; ++j) before += s_img[j] < mine || (s_img[j] == mine && j < i);
        atomicAdd(&s_place[i], before);
    }
    __syncthreads();
    if (t >= n) return;
    const unsigned p = s_place[t];
    st_key<KW>(kout, p, ld_key<KW>(kin, t));
    if (iota) static_cast<int64_t*>(vout)[p] = t;
    else if (vw == 8) static_cast<unsigned long long*>(vout)[p] = __ldg(static_cast<const unsigned long long*>(vin) + t);
    else if (vw == 4) static_cast<unsigned*>(vout)[p] = __ldg(static_cast<const unsigned*>(vin) + t);
}

template <int KW, bool FLT>
__global__ void __launch_bounds__(SM_NT) k_radix_small(const void* __restrict__ kin, const void* __restrict__ vin,
                                                       void* __restrict__ kout, void* __restrict__ vout, int n,
                                                       digit_of<KW, FLT> dg, int end_bit, int vw, int iota) {
    using kt = kreg<KW>;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ unsigned wsum[RS_BINS / 32];
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    unsigned* wh = reinterpret_cast<unsigned*>(smem) + warp * RS_BINS;
    unsigned* wm = reinterpret_cast<unsigned*>(smem) + (SM_WARPS + warp) * RS_BINS;
    unsigned* whd = reinterpret_cast<unsigned*>(smem) + t;
    kt* skeys = reinterpret_cast<kt*>(smem);
    unsigned short* sidx = reinterpret_cast<unsigned short*>(smem + SM_ROWS * sizeof(kt));
    const int ipt = (n + SM_NT - 1) / SM_NT;     // rows per thread
    const int local0 = warp * 32 * ipt + lane;   // row (k, lane) of the warp: local0 + 32 k
    kt key[SM_IPT];
    unsigned idx[SM_IPT], pos[SM_IPT];
#pragma unroll
    for (int k = 0; k < SM_IPT; ++k) {
        idx[k] = local0 + 32 * k;
        key[k] = k < ipt && local0 + 32 * k < n ? ld_key<KW>(kin, local0 + 32 * k) : kt(0);
    }
    for (; dg.shift < end_bit; dg.shift += RS_MAXBITS) {
        dg.mask = (1u << min(RS_MAXBITS, end_bit - dg.shift)) - 1u;
#pragma unroll
        for (int i = 0; i < RS_BINS / 32; i += 4) {
            reinterpret_cast<uint4*>(wh)[i / 4 * 32 + lane] = make_uint4(0, 0, 0, 0);
            reinterpret_cast<uint4*>(wm)[i / 4 * 32 + lane] = make_uint4(0, 0, 0, 0);
        }
        __syncwarp();
#pragma unroll
        for (int k = 0; k < SM_IPT; ++k)
            if (k < ipt) pos[k] = warp_rank(wm, wh, dg(key[k]), local0 + 32 * k < n, lane);
        __syncthreads();
        unsigned tot = 0, incl = 0;
        if (t < RS_BINS) {
#pragma unroll
            for (int w = 0; w < SM_WARPS; ++w) tot += whd[w * RS_BINS];
            incl = dev_::warp_inclusive_sum(tot);
            if (lane == 31) wsum[warp] = incl;
        }
        // One digit in every row: the order stays.
        if (__syncthreads_or(t < RS_BINS && tot == (unsigned)n)) continue;
        if (t < RS_BINS) {
            unsigned run = incl - tot;
            for (int w = 0; w < warp; ++w) run += wsum[w];
#pragma unroll
            for (int w = 0; w < SM_WARPS; ++w) {
                const unsigned c = whd[w * RS_BINS];
                whd[w * RS_BINS] = run;
                run += c;
            }
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < SM_IPT; ++k)
            if (k < ipt && local0 + 32 * k < n) pos[k] += wh[dg(key[k])];
        __syncthreads();
#pragma unroll
        for (int k = 0; k < SM_IPT; ++k)
            if (k < ipt && local0 + 32 * k < n) {
                skeys[pos[k]] = key[k];
                sidx[pos[k]] = (unsigned short)idx[k];
            }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < SM_IPT; ++k)
            if (k < ipt && local0 + 32 * k < n) {
                key[k] = skeys[local0 + 32 * k];
                idx[k] = sidx[local0 + 32 * k];
            }
        __syncthreads();
    }
#pragma unroll
    for (int k = 0; k < SM_IPT; ++k) {
        const int i = local0 + 32 * k;
        if (k >= ipt || i >= n) continue;
        st_key<KW>(kout, i, key[k]);
        if (iota) static_cast<int64_t*>(vout)[i] = idx[k];
        else if (vw == 8) static_cast<unsigned long long*>(vout)[i] = __ldg(static_cast<const unsigned long long*>(vin) + idx[k]);
        else if (vw == 4) static_cast<unsigned*>(vout)[i] = __ldg(static_cast<const unsigned*>(vin) + idx[k]);
    }
}

// Rows per thread of a pass: the most that two CTAs per SM hold, or 4, so that
// a sort of a few thousand to half a million rows spreads over more SMs.  Us a
// call with 4 / the most, int32 keys with int64 values: 2^15 rows 105 / 115,
// 2^18 117 / 124, 3 * 2^17 128 / 125, 2^19 127 / 127, 2^20 163 / 140, 2^22 344 /
// 224; int32 with int32: 2^15 97 / 108, 2^19 121 / 121, 2^20 150 / 124; int64
// with int64: 2^15 135 / 148, 2^18 165 / 163, 2^19 186 / 176, 2^20 252 / 211.
constexpr int OS_IPT_SMALL = 4;
template <int KW, int VW>
int onesweep_ipt(int64_t n) { return n >= (int64_t)1 << 19 ? os_ipt_max<KW, VW>() : OS_IPT_SMALL; }

constexpr int OS_IPT_MIN = os_ipt_max<8, 8>();  // the smallest tile of a large sort
size_t r256(size_t b) { return (b + 255) & ~size_t(255); }
size_t onesweep_temp_bytes(int64_t n, int kw, int vw) {
    return r256((size_t)n * kw) + r256((size_t)n * vw) + r256(sizeof(os_plan)) +
           2 * (size_t)ceil_div(n, (int64_t)OS_NT * (n >= (int64_t)1 << 19 ? OS_IPT_MIN : OS_IPT_SMALL)) * RS_BINS *
               sizeof(os_state);
}

// n > 0, begin_bit < end_bit.  Returns false when a wait gave up
// (the outputs are then unspecified, the inputs untouched).
template <int KW, int VW, bool FLT>
bool onesweep_run(const col& keys, const void* vin, bool iota, const img_params& ip, int begin_bit, int end_bit,
                  void* kout, void* vout, char* tp, cudaStream_t s) {
    const int64_t n = keys.n;
    if (n <= SR_ROWS) {
        k_radix_rank<KW, FLT><<<1, SR_NT, 0, s>>>(keys.data, vin, kout, vout, (int)n,
                                                  make_digit<KW, FLT>(ip, begin_bit, RS_MAXBITS), end_bit - begin_bit,
                                                  VW, iota ? 1 : 0);
        GX_LAUNCHED();
        return true;
    }
    if (n <= SM_ROWS) {
        static per_device_flag attr;
        attr.once([] {
            GX_CUDA(cudaFuncSetAttribute(k_radix_small<KW, FLT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         small_smem<KW>()));
        });
        k_radix_small<KW, FLT><<<1, SM_NT, small_smem<KW>(), s>>>(keys.data, vin, kout, vout, (int)n,
                                                                  make_digit<KW, FLT>(ip, begin_bit, RS_MAXBITS),
                                                                  end_bit, VW, iota ? 1 : 0);
        GX_LAUNCHED();
        return true;
    }
    static per_device_flag attr;
    attr.once([] {
        GX_CUDA(cudaFuncSetAttribute(k_radix_onesweep<KW, VW, FLT, os_ipt_max<KW, VW>()>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, os_smem<KW, VW>(os_ipt_max<KW, VW>())));
        GX_CUDA(cudaFuncSetAttribute(k_radix_onesweep<KW, VW, FLT, OS_IPT_SMALL>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, os_smem<KW, VW>(OS_IPT_SMALL)));
    });
    const int passes = (end_bit - begin_bit + RS_MAXBITS - 1) / RS_MAXBITS;
    const int ipt = onesweep_ipt<KW, VW>(n);
    const int64_t ntiles = ceil_div(n, (int64_t)OS_NT * ipt);
    os_args a;
    a.kin = keys.data;
    a.vin = vin;
    a.kout = kout;
    a.vout = vout;
    a.ktmp = tp;
    tp += r256((size_t)n * KW);
    a.vtmp = tp;
    tp += r256((size_t)n * VW);
    a.n = n;
    a.iota = iota ? 1 : 0;
    a.spin_limit = poll_limit("GX_RADIX_LOOKBACK_POLLS", OS_SPIN_LIMIT);
    a.copy_limit = (uint32_t)poll_limit("GX_RADIX_COPY_POLLS", (int)OS_COPY_WAIT);
    a.plan = reinterpret_cast<os_plan*>(tp);
    tp += r256(sizeof(os_plan));
    a.state[0] = reinterpret_cast<os_state*>(tp);
    a.state[1] = a.state[0] + ntiles * RS_BINS;
    // The first pass needs its own state cleared and clears the other.
    GX_CUDA(cudaMemsetAsync(a.plan, 0, r256(sizeof(os_plan)) + (size_t)ntiles * RS_BINS * sizeof(os_state), s));
    const int hgrid = (int)std::min<int64_t>((int64_t)dev().sm_count * 2, ceil_div(n, (int64_t)OH_NT * 8));
    k_radix_hist_all<KW, FLT><<<hgrid, OH_NT, 0, s>>>(keys.data, n, make_digit<KW, FLT>(ip, 0, RS_MAXBITS), begin_bit,
                                                      end_bit, passes, a.plan);
    GX_LAUNCHED();
    {
        GX_PROF("radix_scatter", s);
        for (int p = 0; p < passes; ++p) {
            const int shift = begin_bit + p * RS_MAXBITS;
            const auto dg = make_digit<KW, FLT>(ip, shift, std::min(RS_MAXBITS, end_bit - shift));
            a.pass = p;
            if (ipt == OS_IPT_SMALL)
                k_radix_onesweep<KW, VW, FLT, OS_IPT_SMALL><<<(unsigned)ntiles, OS_NT, os_smem<KW, VW>(OS_IPT_SMALL), s>>>(dg, a);
            else
                k_radix_onesweep<KW, VW, FLT, os_ipt_max<KW, VW>()>
                    <<<(unsigned)ntiles, OS_NT, os_smem<KW, VW>(os_ipt_max<KW, VW>()), s>>>(dg, a);
            GX_LAUNCHED();
        }
    }
    return read_scalar(&a.plan->err, s) == 0;
}

bool onesweep(const col& keys, const void* vin, int vw, bool iota, const img_params& ip, int begin_bit, int end_bit,
              void* kout, void* vout, char* tp, cudaStream_t s) {
    const bool flt = ip.kind == VK_F;
#define GX_OS_CASE(K, V, F) \
    if (ip.lw == K && vw == V && flt == F) return onesweep_run<K, V, F>(keys, vin, iota, ip, begin_bit, end_bit, kout, vout, tp, s);
#define GX_OS_VALS(K, F) GX_OS_CASE(K, 0, F) GX_OS_CASE(K, 4, F) GX_OS_CASE(K, 8, F)
    GX_OS_VALS(1, false) GX_OS_VALS(2, false) GX_OS_VALS(4, false) GX_OS_VALS(8, false)
    GX_OS_VALS(4, true) GX_OS_VALS(8, true)
#undef GX_OS_VALS
#undef GX_OS_CASE
    fail(GX_EUNSUPPORTED, "radix sort: unsupported key/value width combination");
}

}  // namespace

size_t radix_temp_bytes(int64_t n, int key_width, int val_width) {
    return onesweep_temp_bytes(std::max<int64_t>(n, 1), key_width, val_width) + 256;  // start rounded up to 256
}

void key_image_range(const col& keys, uint64_t* lo, uint64_t* hi, cudaStream_t s) {
    int w = size_of(keys.type);
    require(w == 4 || w == 8, "key_image_range: 4/8-byte keys only");
    img_params ip{vkind_of(keys.type), w, 0, 0};
    dbuf out(16, s);
    GX_CUDA(cudaMemsetAsync(out.get(), 0xFF, 8, s));
    GX_CUDA(cudaMemsetAsync(out.get<char>() + 8, 0, 8, s));
    if (keys.n > 0) {
        int g = grid_for(keys.n, 256, 8);
        if (w == 4) k_image_range<4><<<g, 256, 0, s>>>(keys.data, keys.n, ip, out.get<unsigned long long>());
        else k_image_range<8><<<g, 256, 0, s>>>(keys.data, keys.n, ip, out.get<unsigned long long>());
        GX_LAUNCHED();
    }
    uint64_t h[2];
    host_read(h, out.get(), 16, s);
    *lo = h[0];
    *hi = h[1];
}

// The per-tile passes with their own temporaries (every width, bias).
static void radix_sort_per_tile(const col& keys_c, const void* vals_in, int val_width, bool vals_iota, int begin_bit,
                                int end_bit, const img_params& ip, void* keys_out, void* vals_out, cudaStream_t s) {
    const int64_t n = keys_c.n;
    const int lw = ip.lw;
    // Narrow keys: sort a 32-bit widened copy with the narrow image, then narrow back.
    col keys = keys_c;
    void* kout = keys_out;
    owned_col wide_in;
    dbuf wide_out;
    int kw = lw;
    if (lw < 4) {
        wide_in = widen_to_32(keys_c, s);
        wide_out = dbuf((size_t)n * 4, s);
        keys.data = wide_in.buf.get();
        kout = wide_out.get();
        kw = 4;
    }
    const int passes = (end_bit - begin_bit + RS_MAXBITS - 1) / RS_MAXBITS;
    const int64_t ntiles = ceil_div(n, RS_TILE);
    dbuf tk((size_t)n * kw, s), tv((size_t)n * val_width, s), counts((size_t)RS_BINS * ntiles * 8, s),
        offs((size_t)RS_BINS * ntiles * 8 + 8, s);
    const void* kin = keys.data;
    const void* vin = vals_in;
    bool iota = vals_iota;
    int shift = begin_bit;
    for (int p = 0; p < passes; ++p) {
        int dbits = std::min(RS_MAXBITS, end_bit - shift);
        bool to_out = ((passes - 1 - p) % 2) == 0;
        void* ko = to_out ? kout : tk.get();
        void* vo = to_out ? vals_out : tv.get();
        if (kw == 4) k_radix_hist<4><<<(unsigned)ntiles, RS_NT, 0, s>>>(kin, n, ip, shift, dbits, ntiles, counts.get<int64_t>());
        else k_radix_hist<8><<<(unsigned)ntiles, RS_NT, 0, s>>>(kin, n, ip, shift, dbits, ntiles, counts.get<int64_t>());
        GX_LAUNCHED();
        exclusive_scan_i64(counts.get<int64_t>(), offs.get<int64_t>(), (int64_t(1) << dbits) * ntiles, s);
        scatter_dispatch(kw, val_width, iota, ntiles, s, kin, vin, n, ip, shift, dbits, offs.get<int64_t>(), ko, vo);
        kin = ko;
        vin = vo;
        iota = false;
        shift += dbits;
    }
    if (lw < 4) {
        int g = grid_for(n, 256, 8);
        if (lw == 2) k_narrow<<<g, 256, 0, s>>>((uint16_t*)keys_out, wide_out.get<uint32_t>(), n);
        else k_narrow<<<g, 256, 0, s>>>((uint8_t*)keys_out, wide_out.get<uint32_t>(), n);
        GX_LAUNCHED();
    }
}

// Internal entry with an optional image bias (sort on img - bias).
void radix_sort_biased(const col& keys_c, const void* vals_in, int val_width, bool vals_iota,
                       int begin_bit, int end_bit, bool descending, uint64_t bias, void* keys_out,
                       void* vals_out, void* temp, size_t temp_bytes, cudaStream_t s) {
    const int64_t n = keys_c.n;
    int lw = size_of(keys_c.type);
    require(lw > 0, "radix sort: non-numeric key type " + type_name(keys_c.type));
    require(val_width == 0 || val_width == 4 || val_width == 8 ||
                (val_width > 0 && vals_iota),
            "radix sort: value width must be 0, 4 or 8");
    if (vals_iota) val_width = 8;
    int full = 8 * lw;
    if (end_bit <= 0 || end_bit > full) end_bit = full;
    if (begin_bit < 0) begin_bit = 0;
    if (n == 0) return;

    if (begin_bit >= end_bit) {
        GX_CUDA(cudaMemcpyAsync(keys_out, keys_c.data, (size_t)n * lw, cudaMemcpyDeviceToDevice, s));
        if (val_width) {
            if (vals_iota) sequence_i64(static_cast<int64_t*>(vals_out), n, 0, 1, s);
            else GX_CUDA(cudaMemcpyAsync(vals_out, vals_in, (size_t)n * val_width, cudaMemcpyDeviceToDevice, s));
        }
        return;
    }
    const img_params ip{vkind_of(keys_c.type), lw, descending ? 1 : 0, bias};
    if (!getenv("GX_RADIX_NO_BULK")) {
        dbuf own;
        char* tp = static_cast<char*>(temp);
        if (n > SM_ROWS) {
            if (!tp || temp_bytes < radix_temp_bytes(n, lw, val_width)) {
                own = dbuf(radix_temp_bytes(n, lw, val_width), s);
                tp = own.get<char>();
            }
            tp = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(tp) + 255) & ~uintptr_t(255));
        }
        if (onesweep(keys_c, vals_in, val_width, vals_iota, ip, begin_bit, end_bit, keys_out, vals_out, tp, s)) return;
    }
    radix_sort_per_tile(keys_c, vals_in, val_width, vals_iota, begin_bit, end_bit, ip, keys_out, vals_out, s);
}

void radix_sort(const col& keys, const void* vals_in, int val_width, bool vals_iota, int begin_bit,
                int end_bit, bool descending, void* keys_out, void* vals_out, void* temp,
                size_t temp_bytes, cudaStream_t s) {
    radix_sort_biased(keys, vals_in, val_width, vals_iota, begin_bit, end_bit, descending, 0,
                      keys_out, vals_out, temp, temp_bytes, s);
}

}  // namespace gx

namespace gx {

// Scratch bytes radix_sort_pairs_scratch needs for n pairs of 4/8-byte keys
// and 4/8-byte values: both ping-pong halves, the per-tile digit counts and
// offsets, and the scan's temporaries (each rounded to 256 bytes).
size_t radix_pairs_scratch_bytes(int64_t n, int key_width, int val_width) {
    auto r256 = [](size_t b) { return (b + 255) & ~size_t(255); };
    int64_t ntiles = ceil_div(std::max<int64_t>(n, 1), RS_TILE);
    size_t b = r256((size_t)n * key_width) + r256((size_t)n * val_width);
    b += r256((size_t)RS_BINS * ntiles * 8) + r256((size_t)RS_BINS * ntiles * 8 + 8);
    return b + scan_scratch_bytes((int64_t)RS_BINS * ntiles);
}

// Raises the dynamic shared-memory limit of every 4/8-byte (key, value)
// scatter instantiation on the current device, so later pair sorts of any
// width combination launch without changing a kernel attribute.
void radix_prepare_pair_scatters() {
    prepare_scatter<4, 4, false>();
    prepare_scatter<4, 8, false>();
    prepare_scatter<8, 4, false>();
    prepare_scatter<8, 8, false>();
}

// The pass loop of radix_sort_biased (bias 0) for 4/8-byte keys and values,
// with every temporary taken from `scratch`.  The histogram and scatter
// kernels are the same, so the output equals gx_sort_column_pair's.  The
// caller has checked key/value widths and that scratch holds
// radix_pairs_scratch_bytes(n, kw, vw).  Nothing in scratch is read before
// it is written in the same call.
void radix_sort_pairs_scratch(const col& keys, const void* vals_in, int val_width, int begin_bit, int end_bit,
                              bool descending, void* keys_out, void* vals_out, char* scratch, cudaStream_t s) {
    const int64_t n = keys.n;
    const int kw = size_of(keys.type);
    int full = 8 * kw;
    if (end_bit <= 0 || end_bit > full) end_bit = full;
    if (begin_bit < 0) begin_bit = 0;
    if (n == 0) return;
    auto take = [&](size_t bytes) {
        char* p = scratch;
        scratch += (bytes + 255) & ~size_t(255);
        return p;
    };
    img_params ip{vkind_of(keys.type), kw, descending ? 1 : 0, 0};
    int nbits = end_bit - begin_bit;
    int passes = nbits > 0 ? (nbits + RS_MAXBITS - 1) / RS_MAXBITS : 0;
    if (passes == 0) {
        GX_CUDA(cudaMemcpyAsync(keys_out, keys.data, (size_t)n * kw, cudaMemcpyDeviceToDevice, s));
        GX_CUDA(cudaMemcpyAsync(vals_out, vals_in, (size_t)n * val_width, cudaMemcpyDeviceToDevice, s));
        return;
    }
    int64_t ntiles = ceil_div(n, RS_TILE);
    char* tk = take((size_t)n * kw);
    char* tv = take((size_t)n * val_width);
    int64_t* counts = reinterpret_cast<int64_t*>(take((size_t)RS_BINS * ntiles * 8));
    int64_t* offs = reinterpret_cast<int64_t*>(take((size_t)RS_BINS * ntiles * 8 + 8));
    char* scan_tmp = scratch;
    const void* kin = keys.data;
    const void* vin = vals_in;
    int shift = begin_bit;
    for (int p = 0; p < passes; ++p) {
        int dbits = std::min(RS_MAXBITS, end_bit - shift);
        bool to_out = ((passes - 1 - p) % 2) == 0;
        void* ko = to_out ? keys_out : tk;
        void* vo = to_out ? vals_out : tv;
        if (kw == 4) k_radix_hist<4><<<(unsigned)ntiles, RS_NT, 0, s>>>(kin, n, ip, shift, dbits, ntiles, counts);
        else k_radix_hist<8><<<(unsigned)ntiles, RS_NT, 0, s>>>(kin, n, ip, shift, dbits, ntiles, counts);
        GX_LAUNCHED();
        int64_t bins = 1 << dbits;
        exclusive_scan_i64_scratch(counts, offs, bins * ntiles, scan_tmp, s);
        scatter_dispatch(kw, val_width, false, ntiles, s, kin, vin, n, ip, shift, dbits, offs, ko, vo);
        kin = ko;
        vin = vo;
        shift += dbits;
    }
}

}  // namespace gx
