// gx_dict.cu — dictionary encoding.
//
// Replaces gamax::compress::dictionary_encode{,_with_order} and the
// ready-dictionary overload (src/cuda/compress/dictionary_encode.cu:144-373,
// src/cuda/compress/dictionary_encode_dict_ready.cu:16-82).  The reference
// inserts row ids into a cuco set sized N/0.25 when no hint is given, writes
// an int64 representative per row and gathers codes through it.  Here a table
// slot holds the canonical key bits and their code side by side, so one access
// yields both:
//   * hash encode: one pass that inserts keys, hands each new key the next
//     code (atomicAdd) and writes every row's code;
//   * order-preserving: the same pass writes first-insert codes and lists the
//     distinct keys in that order; the keys are radix-sorted and a second pass
//     replaces each code by its key's rank (a gather from ndv entries instead
//     of another table lookup);
//   * ready dictionary: the dictionary's values are inserted with code =
//     position (the smallest position wins for duplicated values); rows whose
//     value is absent get INT32_MIN (gamax::sentinel<int32_t>()).
// Without a size hint the table is sized from a HyperLogLog estimate
// instead of the row count.
#include <algorithm>
#include <cmath>

#include "gx_groupby.h"

namespace gx {
namespace {

// Slots.  4-byte keys: one word, key << 32 | code.  8-byte keys: a 16-byte
// pair {key, code}.  All bits set is an empty slot in both, so one memset
// clears a table; the 8-byte key of all ones lives in the extra slot `cap`,
// told apart by its code alone.
constexpr unsigned long long D_EMPTY = ~0ull;
constexpr uint64_t NO_CODE = ~0ull;                 // key absent
constexpr uint64_t PENDING = ~0ull - 1;             // key claimed, code not yet there
constexpr uint32_t PENDING4 = 0xFFFFFFFEu;
constexpr uint32_t D_WAIT_LIMIT = 1u << 16;

struct dtable {
    unsigned long long* w;
    uint64_t mask;
    int* overflow;
};

template <int KW>
__device__ __forceinline__ uint64_t dkey(const void* p, int64_t i, int kind) {
    if (KW == 4) return canon32(__ldg(static_cast<const unsigned*>(p) + i), kind);
    return canon64(__ldg(static_cast<const unsigned long long*>(p) + i), kind);
}
template <int KW>
__device__ __forceinline__ uint64_t dhash(uint64_t k) {
    if (KW == 4) return fmix32((uint32_t)k);
    return fmix64(k);
}

// Code of key k when it sits, settled, in its home slot (one plain load),
// else NO_CODE: a stale read only sends the row to the full walk.
template <int KW>
__device__ __forceinline__ uint64_t d_home(const dtable& t, uint64_t k) {
    const uint64_t slot = dhash<KW>(k) & t.mask;
    if constexpr (KW == 4) {
        const unsigned long long c = t.w[slot];
        return (uint32_t)(c >> 32) == (uint32_t)k && (uint32_t)c < PENDING4 ? (uint64_t)(uint32_t)c : NO_CODE;
    } else {
        const ulonglong2 c = reinterpret_cast<const ulonglong2*>(t.w)[slot];
        return c.x == k && k != D_EMPTY && c.y < PENDING ? c.y : NO_CODE;
    }
}

// Hands out the next code and lists its key.
__device__ __forceinline__ uint64_t d_next(unsigned long long* counter, void* dkeys, int kw, uint64_t k) {
    const unsigned long long c = atomicAdd(counter, 1ull);
    if (dkeys) {
        if (kw == 4) static_cast<unsigned*>(dkeys)[c] = (unsigned)k;
        else static_cast<unsigned long long*>(dkeys)[c] = k;
    }
    return c;
}

// Code of key k, inserting it.  PENDING when another thread has claimed the
// key and not yet published its code (the inserter may be a lane of the same
// warp, which a spinning branch could hold back); NO_CODE when the walk ran
// out (overflow set).
template <int KW>
__device__ __forceinline__ uint64_t d_insert(const dtable& t, uint64_t k, unsigned long long* counter, void* dkeys) {
    if (KW == 8 && k == D_EMPTY) {
        unsigned long long* code = t.w + 2 * (t.mask + 1) + 1;
        unsigned long long c = *(volatile unsigned long long*)code;
        if (c != NO_CODE) return c;
        c = atomicCAS(code, NO_CODE, PENDING);
        if (c != NO_CODE) return c;
        c = d_next(counter, dkeys, KW, k);
        *(volatile unsigned long long*)code = c;
        return c;
    }
    uint64_t slot = dhash<KW>(k) & t.mask;
    for (uint64_t p = 0, lim = t.mask < GX_PROBE_LIMIT ? t.mask : GX_PROBE_LIMIT - 1; p <= lim; ++p) {
        if constexpr (KW == 4) {
            unsigned long long cur = ((volatile unsigned long long*)t.w)[slot];
            if (cur == D_EMPTY) {
                cur = atomicCAS(&t.w[slot], D_EMPTY, (unsigned long long)k << 32 | PENDING4);
                if (cur == D_EMPTY) {
                    const uint64_t c = d_next(counter, dkeys, KW, k);
                    ((volatile unsigned long long*)t.w)[slot] = (unsigned long long)k << 32 | (uint32_t)c;
                    return c;
                }
            }
            if ((uint32_t)(cur >> 32) == (uint32_t)k) return (uint32_t)cur == PENDING4 ? PENDING : (uint64_t)(uint32_t)cur;
        } else {
            unsigned long long* s = t.w + 2 * slot;
            unsigned long long cur = *(volatile unsigned long long*)s;
            if (cur == D_EMPTY) {
                cur = atomicCAS(s, D_EMPTY, (unsigned long long)k);
                if (cur == D_EMPTY) {
                    const uint64_t c = d_next(counter, dkeys, KW, k);
                    ((volatile unsigned long long*)s)[1] = c;
                    return c;
                }
            }
            if (cur == k) {
                const unsigned long long c = ((volatile unsigned long long*)s)[1];
                return c == NO_CODE ? PENDING : c;
            }
        }
        slot = (slot + 1) & t.mask;
    }
    atomicExch(t.overflow, 1);
    return NO_CODE;
}

// Code of key k in a finished table, NO_CODE when absent.
template <int KW>
__device__ __forceinline__ uint64_t d_find(const dtable& t, uint64_t k) {
    if (KW == 8 && k == D_EMPTY) return t.w[2 * (t.mask + 1) + 1];
    uint64_t slot = dhash<KW>(k) & t.mask;
    for (uint64_t p = 0, lim = t.mask < GX_PROBE_LIMIT ? t.mask : GX_PROBE_LIMIT - 1; p <= lim; ++p) {
        if constexpr (KW == 4) {
            const unsigned long long cur = t.w[slot];
            if (cur == D_EMPTY) return NO_CODE;
            if ((uint32_t)(cur >> 32) == (uint32_t)k) return (uint32_t)cur;
        } else {
            const ulonglong2 cur = reinterpret_cast<const ulonglong2*>(t.w)[slot];
            if (cur.x == D_EMPTY) return NO_CODE;
            if (cur.x == k) return cur.y;
        }
        slot = (slot + 1) & t.mask;
    }
    return NO_CODE;
}

__device__ __forceinline__ void store_code(void* out, int w, int64_t i, uint64_t c) {
    switch (w) {
        case 8: static_cast<unsigned long long*>(out)[i] = c; break;
        case 4: static_cast<unsigned*>(out)[i] = (unsigned)c; break;
        case 2: static_cast<uint16_t*>(out)[i] = (uint16_t)c; break;
        default: static_cast<uint8_t*>(out)[i] = (uint8_t)c; break;
    }
}

// Rows per thread per round: their keys are loaded, then their home slots
// read, all at once, so each thread keeps DU independent table reads in
// flight instead of one dependent chain.
constexpr int DU = 4;
constexpr int D_NT = 256;

// Inserts every row's key and writes its code.  Bound by one random L2 sector
// per row; rows displaced from their home slot (an eighth at load 1/4) are
// queued per warp and walk the table 32 at a time.  Order-preserving codes of
// 10^8 int32 rows with 2^16 values: 1.18 ms a call, 1.44 when each row walked by
// itself, 1.81 with a key table and a code table read in two passes.
template <int KW>
__global__ void __launch_bounds__(D_NT) k_dict_encode(const void* __restrict__ keys, int64_t n, int kind, dtable t,
                                                      unsigned long long* __restrict__ counter,
                                                      void* __restrict__ dkeys, void* __restrict__ out, int ow) {
    __shared__ int64_t s_q[D_NT / 32][31 + 32 * DU];  // rows of a warp that are not settled in their home slot
    int64_t* queue = s_q[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    int fill = 0;
    // Walks the table for the last m <= 32 queued rows, a lane each; rows that
    // meet a pending code are tried again after the warp has regrouped.
    auto walk = [&](int m) {
        fill -= m;
        const bool live = lane < m;
        const int64_t i = live ? queue[fill + lane] : 0;
        const uint64_t k = live ? dkey<KW>(keys, i, kind) : 0;
        uint64_t c = live ? d_insert<KW>(t, k, counter, dkeys) : 0;
        for (uint32_t round = 0; __any_sync(0xffffffffu, c == PENDING); ++round) {
            __syncwarp();
            if (c != PENDING) continue;
            if (round < D_WAIT_LIMIT) c = d_insert<KW>(t, k, counter, dkeys);
            else {
                atomicExch(t.overflow, 1);
                c = NO_CODE;
            }
        }
        if (live) store_code(out, ow, i, c);
        __syncwarp();
    };
    const int64_t step = (int64_t)gridDim.x * D_NT;
    const int64_t rounds = (n + step * DU - 1) / (step * DU);  // whole warps stay in the loop together
    for (int64_t r = 0; r < rounds; ++r) {
        const int64_t i0 = r * step * DU + blockIdx.x * (int64_t)D_NT + threadIdx.x;
        uint64_t k[DU], c[DU];
#pragma unroll
        for (int q = 0; q < DU; ++q) k[q] = i0 + q * step < n ? dkey<KW>(keys, i0 + q * step, kind) : 0;
#pragma unroll
        for (int q = 0; q < DU; ++q) c[q] = i0 + q * step < n ? d_home<KW>(t, k[q]) : 0;
#pragma unroll
        for (int q = 0; q < DU; ++q) {
            const bool valid = i0 + q * step < n, miss = valid && c[q] == NO_CODE;
            const unsigned m = __ballot_sync(0xffffffffu, miss);
            if (miss) queue[fill + __popc(m & ((1u << lane) - 1u))] = i0 + q * step;
            fill += __popc(m);
            if (valid && !miss) store_code(out, ow, i0 + q * step, c[q]);
        }
        __syncwarp();
        while (fill >= 32) walk(32);
    }
    walk(fill);
}

// Replaces first-insert codes by ranks: out[i] = rank[code[i]].
template <typename T>
__global__ void __launch_bounds__(D_NT) k_dict_remap(const T* codes, int64_t n,
                                                     const T* __restrict__ rank, void* out, int ow) {
    const int64_t step = (int64_t)gridDim.x * D_NT;
    for (int64_t i0 = blockIdx.x * (int64_t)D_NT + threadIdx.x; i0 < n; i0 += step * DU) {
        T c[DU];
#pragma unroll
        for (int q = 0; q < DU; ++q) c[q] = i0 + q * step < n ? codes[i0 + q * step] : T(0);
#pragma unroll
        for (int q = 0; q < DU; ++q) c[q] = __ldg(rank + c[q]);
#pragma unroll
        for (int q = 0; q < DU; ++q)
            if (i0 + q * step < n) store_code(out, ow, i0 + q * step, c[q]);
    }
}
template <typename T>
__global__ void k_dict_rank(const int64_t* __restrict__ sorted_src, int64_t m, T* __restrict__ rank) {
    for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < m; r += (int64_t)gridDim.x * blockDim.x)
        rank[sorted_src[r]] = (T)r;
}

// Ready dictionary: insert value -> smallest position.
template <int KW>
__global__ void k_dict_insert_positions(const void* __restrict__ dict, int64_t n, int kind, dtable t) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const uint64_t k = dkey<KW>(dict, i, kind);
        if (KW == 8 && k == D_EMPTY) {
            atomicMin(t.w + 2 * (t.mask + 1) + 1, (unsigned long long)i);
            continue;
        }
        const unsigned long long word = (unsigned long long)k << 32 | (uint32_t)min(i, (int64_t)PENDING4 - 1);
        uint64_t slot = dhash<KW>(k) & t.mask;
        bool done = false;
        for (uint64_t p = 0, lim = t.mask < GX_PROBE_LIMIT ? t.mask : GX_PROBE_LIMIT - 1; p <= lim && !done; ++p) {
            if constexpr (KW == 4) {
                unsigned long long cur = ((volatile unsigned long long*)t.w)[slot];
                if (cur == D_EMPTY) cur = atomicCAS(&t.w[slot], D_EMPTY, word);
                if (cur == D_EMPTY) done = true;
                else if ((uint32_t)(cur >> 32) == (uint32_t)k) {
                    atomicMin(&t.w[slot], word);  // same key: the smaller position
                    done = true;
                }
            } else {
                unsigned long long* s = t.w + 2 * slot;
                unsigned long long cur = *(volatile unsigned long long*)s;
                if (cur == D_EMPTY) cur = atomicCAS(s, D_EMPTY, (unsigned long long)k);
                if (cur == D_EMPTY || cur == k) {
                    atomicMin(s + 1, (unsigned long long)i);
                    done = true;
                }
            }
            slot = (slot + 1) & t.mask;
        }
        if (!done) atomicExch(t.overflow, 1);
    }
}

template <int KW>
__global__ void __launch_bounds__(D_NT) k_dict_lookup(const void* __restrict__ keys, int64_t n, int kind, dtable t,
                                                      void* __restrict__ out, int ow, uint64_t missing) {
    const int64_t step = (int64_t)gridDim.x * D_NT;
    for (int64_t i0 = blockIdx.x * (int64_t)D_NT + threadIdx.x; i0 < n; i0 += step * DU) {
        uint64_t k[DU], c[DU];
#pragma unroll
        for (int q = 0; q < DU; ++q) k[q] = i0 + q * step < n ? dkey<KW>(keys, i0 + q * step, kind) : 0;
#pragma unroll
        for (int q = 0; q < DU; ++q) c[q] = i0 + q * step < n ? d_home<KW>(t, k[q]) : 0;
#pragma unroll
        for (int q = 0; q < DU; ++q)
            if (c[q] == NO_CODE) c[q] = d_find<KW>(t, k[q]);
#pragma unroll
        for (int q = 0; q < DU; ++q)
            if (i0 + q * step < n) store_code(out, ow, i0 + q * step, c[q] == NO_CODE ? missing : c[q]);
    }
}

struct table_bufs {
    dbuf slots, flags;  // flags: overflow, then the code counter
    dtable t;
};

table_bufs make_table(int64_t cap, int kw, cudaStream_t s) {
    table_bufs b;
    const size_t bytes = (size_t)(cap + 1) * (kw == 4 ? 8 : 16);
    b.slots = dbuf(bytes, s);
    b.flags = dbuf(16, s);
    GX_CUDA(cudaMemsetAsync(b.slots.get(), 0xFF, bytes, s));
    GX_CUDA(cudaMemsetAsync(b.flags.get(), 0, 16, s));
    b.t.w = b.slots.get<unsigned long long>();
    b.t.mask = (uint64_t)cap - 1;
    b.t.overflow = b.flags.get<int>();
    return b;
}

col widen_if_narrow(const col& c, owned_col& hold, cudaStream_t s) {
    if (size_of(c.type) >= 4) return c;
    hold = widen_to_32(c, s);
    col w = c;
    w.data = hold.buf.get();
    w.type = hold.type;
    return w;
}

void check_encode(const col& c, int encode_type) {
    if (c.type == GX_STRING) fail(GX_EINVAL, "Cannot dictionary encode column of type STRING");
    require(is_numeric(c.type), "dictionary encode: unsupported column type " + type_name(c.type));
    if (!(is_signed_int(encode_type) || is_unsigned_int(encode_type)))
        fail(GX_EINVAL, "Encoded type must be integral, got " + type_name(encode_type));
}

int64_t table_capacity(const col& key, int64_t hint, double load_factor, cudaStream_t s) {
    int64_t est;
    if (hint > 0) est = hint;
    else if (key.n <= (1 << 16)) est = key.n;
    else est = std::min<int64_t>(key.n, ndv_estimate(key, s) * 9 / 8 + 64);
    double lf = load_factor > 0.05 && load_factor < 0.95 ? load_factor : 0.25;
    if (lf < 0.5 && est > (1 << 22)) lf = 0.5;  // keep very large tables compact
    return (int64_t)next_pow2((uint64_t)std::max<double>(64.0, std::ceil((double)est / lf)));
}

}  // namespace

// mode: 0 = hash codes, 1 = order-preserving codes.
void dictionary_encode(const gx_column_view& v, int encode_type, int64_t size_hint, double load_factor, int mode,
                       cudaStream_t s, gx_column* out, int64_t* dict_size) {
    col c0 = resolve(v);
    check_encode(c0, encode_type);
    owned_col hold;
    col c = widen_if_narrow(c0, hold, s);
    const int kw = size_of(c.type);
    const int kind = vkind_of(c.type);
    const int ow = size_of(encode_type);
    owned_col res = make_col(encode_type, c.n, s);
    int64_t cap = table_capacity(c, size_hint, load_factor, s);
    // Order-preserving codes start as first-insert codes, in the result itself
    // when it is wide enough.
    dbuf narrow;
    void* first = res.buf.get();
    const int fw = mode == 1 && ow < 4 ? 4 : ow;
    if (fw != ow) {
        narrow = dbuf((size_t)c.n * fw, s);
        first = narrow.get();
    }
    for (int attempt = 0; attempt < 6; ++attempt, cap *= 4) {
        table_bufs tb = make_table(cap, kw, s);
        unsigned long long* counter = reinterpret_cast<unsigned long long*>(tb.flags.get<char>() + 8);
        dbuf dk;  // distinct keys in code order
        if (mode == 1) dk = dbuf((size_t)std::min<int64_t>(cap + 1, std::max<int64_t>(c.n, 1)) * kw, s);
        int g = grid_for(c.n, D_NT, 8);
        if (c.n > 0) {
            GX_PROF("dict_insert", s);
            if (kw == 4) k_dict_encode<4><<<g, D_NT, 0, s>>>(c.data, c.n, kind, tb.t, counter, dk.get(), first, fw);
            else k_dict_encode<8><<<g, D_NT, 0, s>>>(c.data, c.n, kind, tb.t, counter, dk.get(), first, fw);
            GX_LAUNCHED();
        }
        int hflags[4];
        host_read(hflags, tb.flags.get(), 16, s);
        if (hflags[0]) continue;
        unsigned long long ndv_u;
        std::memcpy(&ndv_u, &hflags[2], 8);
        int64_t ndv = (int64_t)ndv_u;
        if (mode == 1 && ndv > 0) {
            // Sort the distinct keys (with their codes) in value order.
            col kc;
            kc.data = dk.get();
            kc.n = ndv;
            kc.type = c.type;
            dbuf sk((size_t)ndv * kw, s), si((size_t)ndv * 8, s), rank((size_t)ndv * fw, s);
            radix_sort(kc, nullptr, 8, true, 0, -1, false, sk.get(), si.get(), nullptr, 0, s);
            const int rg = grid_for(ndv, 256, 8);
            GX_PROF("dict_lookup", s);
            if (fw == 8) {
                k_dict_rank<<<rg, 256, 0, s>>>(si.get<int64_t>(), ndv, rank.get<unsigned long long>());
                GX_LAUNCHED();
                k_dict_remap<<<g, D_NT, 0, s>>>(static_cast<const unsigned long long*>(first), c.n,
                                               rank.get<unsigned long long>(), res.buf.get(), ow);
            } else {
                k_dict_rank<<<rg, 256, 0, s>>>(si.get<int64_t>(), ndv, rank.get<unsigned>());
                GX_LAUNCHED();
                k_dict_remap<<<g, D_NT, 0, s>>>(static_cast<const unsigned*>(first), c.n, rank.get<unsigned>(),
                                               res.buf.get(), ow);
            }
            GX_LAUNCHED();
            GX_CUDA(cudaStreamSynchronize(s));
        }
        *dict_size = ndv;
        *out = to_gx_column(std::move(res));
        return;
    }
    fail(GX_EOVERFLOW, "dictionary table overflow after retries");
}

void dictionary_encode_with_dict(const gx_column_view& v, const gx_column_view& dv, int encode_type, cudaStream_t s,
                                 gx_column* out) {
    col c0 = resolve(v), d0 = resolve(dv);
    if (encode_type != GX_INT32) fail(GX_EINVAL, "Unsupported encoded type");
    require(is_numeric(c0.type), "Dictionary encoding is not supported for non-integral type.");
    require(c0.type == d0.type, "dictionary encode: dictionary type differs from column type");
    owned_col h1, h2;
    col c = widen_if_narrow(c0, h1, s), d = widen_if_narrow(d0, h2, s);
    const int kw = size_of(c.type);
    const int kind = vkind_of(c.type);
    owned_col res = make_col(GX_INT32, c.n, s);
    // The reference sizes its map at dict.size() / 0.3 (dictionary_encode_dict_ready.cu:35-36).
    int64_t cap = (int64_t)next_pow2((uint64_t)std::max<double>(64.0, std::ceil(d.n / 0.3)));
    for (int attempt = 0; attempt < 6; ++attempt, cap *= 4) {
        table_bufs tb = make_table(cap, kw, s);
        if (d.n > 0) {
            int g = grid_for(d.n, 256, 8);
            if (kw == 4) k_dict_insert_positions<4><<<g, 256, 0, s>>>(d.data, d.n, kind, tb.t);
            else k_dict_insert_positions<8><<<g, 256, 0, s>>>(d.data, d.n, kind, tb.t);
            GX_LAUNCHED();
        }
        int ovf = read_scalar(tb.flags.get<int>(), s);
        if (ovf) continue;
        if (c.n > 0) {
            int g = grid_for(c.n, D_NT, 8);
            uint64_t missing = (uint64_t)(uint32_t)0x80000000u;
            if (kw == 4) k_dict_lookup<4><<<g, D_NT, 0, s>>>(c.data, c.n, kind, tb.t, res.buf.get(), 4, missing);
            else k_dict_lookup<8><<<g, D_NT, 0, s>>>(c.data, c.n, kind, tb.t, res.buf.get(), 4, missing);
            GX_LAUNCHED();
        }
        GX_CUDA(cudaStreamSynchronize(s));
        *out = to_gx_column(std::move(res));
        return;
    }
    fail(GX_EOVERFLOW, "dictionary table overflow after retries");
}

}  // namespace gx
