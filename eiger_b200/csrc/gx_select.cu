// gx_select.cu — filter: predicate -> BOOL8 mask -> order-preserving
// compaction, and the fused form that evaluates the predicate while
// compacting.
//
// Replaces gamax::select::select_to_bitmask / select (src/cuda/operators/
// select/select.hpp:15-64, select.cu:19-60) for predicates that are a
// conjunction or disjunction of comparisons of a column with literals, and
// gamax::util::device::compact / count_nonzero (src/cuda/utils/transform.hpp:
// 34-48, transform.cu:74-95,147-205: cub::DeviceSelect::Flagged per column
// plus a thrust reduction of the mask).  The reference's general expression
// trees (expr/expr_fast.hpp) are outside this library.
//
// B200 design: rows are taken in 4096-row tiles (256 threads x 16 rows, the
// rows of a warp contiguous).  k_sel_bits evaluates the predicates once, one
// column at a time with a thread's 16 loads issued together, and writes one
// bit per row and each tile's kept-row count; an exclusive scan places the
// tiles; k_sel_write ranks the kept rows from the bits alone (no barrier, no
// second evaluation) and copies every column's kept values to consecutive
// positions, eight loads in flight per thread, in input order (the order
// cub::DeviceSelect keeps).
#include <cmath>
#include <limits>
#include <type_traits>

#include "gx_groupby.h"

namespace gx {
namespace {

constexpr int SL_NT = 256;
constexpr int SL_IPT = 16;
constexpr int SL_TILE = SL_NT * SL_IPT;
constexpr int MAX_PRED = 8;
constexpr int MAX_SEL_COLS = 32;

// A predicate as a closed range of its column's own type: LT, LE, GT, GE, EQ,
// NE and BETWEEN all become lo <= x <= hi, negated for NE; an empty range
// (nothing compares true) is lo = 1, hi = 0.  NaN lies in no range, so it
// passes NE only, as in the comparisons themselves.
struct pred_dev {
    int n;
    int combine;  // 0 = AND, 1 = OR
    const void* data[MAX_PRED];
    int type[MAX_PRED];
    int negate[MAX_PRED];
    uint64_t lo[MAX_PRED], hi[MAX_PRED];  // bits of the bounds, widened to int64 / uint64 / double
};

struct sel_cols {
    int n;
    const void* in[MAX_SEL_COLS];
    void* out[MAX_SEL_COLS];
    int width[MAX_SEL_COLS];
};

template <class T>
__device__ __forceinline__ T bound_of(uint64_t bits) {
    if constexpr (std::is_floating_point<T>::value) return (T)__longlong_as_double((long long)bits);
    else return (T)bits;
}

// Bit k: row row0 + 32 k is in the range of predicate j, for the rows of `need`
// (no other is read).  float32 values are compared as doubles: the literal
// need not be a float.
template <class T>
__device__ __forceinline__ unsigned range_bits(const pred_dev& p, int j, int64_t row0, unsigned need) {
    using C = typename std::conditional<std::is_same<T, float>::value, double, T>::type;
    const T* d = static_cast<const T*>(p.data[j]);
    const C lo = bound_of<C>(p.lo[j]), hi = bound_of<C>(p.hi[j]);
    T x[SL_IPT];
#pragma unroll
    for (int k = 0; k < SL_IPT; ++k) x[k] = (need >> k) & 1u ? __ldg(d + row0 + k * 32) : T(0);
    unsigned b = 0;
#pragma unroll
    for (int k = 0; k < SL_IPT; ++k) b |= ((C)x[k] >= lo && (C)x[k] <= hi ? 1u : 0u) << k;
    return p.negate[j] ? ~b : b;
}

// Whole warps.  A predicate after the first reads only rows that it decides
// (AND: kept so far, OR: not yet), and none when a warp has no such row.  2^26
// rows, eight 8-byte columns under AND, the first predicate true for 1 in 10^5
// rows: 200 us a call, 710 when every predicate read every row.
__device__ __forceinline__ unsigned keep_bits(const pred_dev& p, int64_t row0, int64_t n) {
    const int64_t rows = (n - row0 + 31) >> 5;  // of this thread, below n
    const unsigned valid = rows >= SL_IPT ? (1u << SL_IPT) - 1u : rows <= 0 ? 0u : (1u << rows) - 1u;
    unsigned keep = p.combine == 0 ? valid : 0u;
    for (int j = 0; j < p.n; ++j) {
        const unsigned need = p.combine == 0 ? keep : valid & ~keep;
        if (!__any_sync(0xffffffffu, need)) break;
        unsigned b;
        switch (p.type[j]) {
            case GX_INT8: b = range_bits<signed char>(p, j, row0, need); break;
            case GX_INT16: b = range_bits<short>(p, j, row0, need); break;
            case GX_INT32: b = range_bits<int>(p, j, row0, need); break;
            case GX_INT64: b = range_bits<long long>(p, j, row0, need); break;
            case GX_UINT16: b = range_bits<unsigned short>(p, j, row0, need); break;
            case GX_UINT32: b = range_bits<unsigned>(p, j, row0, need); break;
            case GX_UINT64: b = range_bits<unsigned long long>(p, j, row0, need); break;
            case GX_FLOAT32: b = range_bits<float>(p, j, row0, need); break;
            case GX_FLOAT64: b = range_bits<double>(p, j, row0, need); break;
            default: b = range_bits<unsigned char>(p, j, row0, need); break;  // UINT8, BOOL8
        }
        keep = p.combine == 0 ? keep & b : keep | (need & b);
    }
    return keep;
}

// Row (k, lane) of warp w in tile t: t*TILE + w*32*IPT + k*32 + lane.
__global__ void __launch_bounds__(SL_NT) k_sel_mask(pred_dev p, int64_t n, uint8_t* __restrict__ out) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t row0 = blockIdx.x * (int64_t)SL_TILE + warp * 32 * SL_IPT + lane;
    const unsigned keep = keep_bits(p, row0, n);
#pragma unroll
    for (int k = 0; k < SL_IPT; ++k)
        if (row0 + k * 32 < n) out[row0 + k * 32] = (keep >> k) & 1u;
}

// bits (when given): word i holds rows 32 i .. 32 i + 31, SL_TILE / 32 words a
// tile.  Bound by HBM.
__global__ void __launch_bounds__(SL_NT) k_sel_bits(pred_dev p, int64_t n, unsigned* __restrict__ bits,
                                                    int64_t* __restrict__ tile_cnt) {
    __shared__ int sm[SL_NT / 32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t row0 = blockIdx.x * (int64_t)SL_TILE + warp * 32 * SL_IPT + lane;
    const unsigned keep = keep_bits(p, row0, n);
    if (bits) {
        unsigned mine = 0;
#pragma unroll
        for (int k = 0; k < SL_IPT; ++k) {
            const unsigned w = __ballot_sync(0xffffffffu, (keep >> k) & 1u);
            if (lane == k) mine = w;
        }
        if (lane < SL_IPT) bits[(blockIdx.x * (int64_t)(SL_NT / 32) + warp) * SL_IPT + lane] = mine;
    }
    const int c = dev_::warp_sum(__popc(keep));
    if (lane == 0) sm[warp] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        int64_t t = 0;
        for (int w = 0; w < SL_NT / 32; ++w) t += sm[w];
        tile_cnt[blockIdx.x] = t;
    }
}

// Copies the kept rows of one column: eight loads in flight per thread.  `at`
// is the first kept row's position of this warp, word[k] the bits of its rows
// 32 k .. 32 k + 31.
template <class T>
__device__ __forceinline__ void copy_kept(const void* in, void* out, int64_t row0, int64_t at, unsigned mine,
                                          unsigned lt, int lane) {
    const T* src = static_cast<const T*>(in) + row0;
    T* dst = static_cast<T*>(out);
    constexpr int B = 8;
#pragma unroll
    for (int k0 = 0; k0 < SL_IPT; k0 += B) {
        T x[B];
        unsigned w[B];
#pragma unroll
        for (int q = 0; q < B; ++q) {
            w[q] = __shfl_sync(0xffffffffu, mine, k0 + q);
            if ((w[q] >> lane) & 1u) x[q] = __ldg(src + (k0 + q) * 32);
        }
#pragma unroll
        for (int q = 0; q < B; ++q) {
            if ((w[q] >> lane) & 1u) dst[at + __popc(w[q] & lt)] = x[q];
            at += __popc(w[q]);
        }
    }
}

// Bound by HBM; see the figures at compact_rows.
__global__ void __launch_bounds__(SL_NT) k_sel_write(const unsigned* __restrict__ bits,
                                                     const int64_t* __restrict__ tile_off, sel_cols c) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t row0 = blockIdx.x * (int64_t)SL_TILE + warp * 32 * SL_IPT + lane;
    constexpr int WORDS = SL_TILE / 32;  // of a tile; lane l counts words 4 l .. 4 l + 3
    static_assert(WORDS == 128 && SL_IPT == 16, "a warp's bits are the words of four lanes");
    const unsigned* tb = bits + blockIdx.x * (int64_t)WORDS;
    const uint4 q = __ldg(reinterpret_cast<const uint4*>(tb) + lane);
    const int before = lane < warp * 4 ? __popc(q.x) + __popc(q.y) + __popc(q.z) + __popc(q.w) : 0;
    const int64_t at = tile_off[blockIdx.x] + dev_::warp_sum(before);
    const unsigned mine = __ldg(tb + warp * SL_IPT + (lane & (SL_IPT - 1)));
    if (!__any_sync(0xffffffffu, mine)) return;
    const unsigned lt = (1u << lane) - 1u;
    for (int j = 0; j < c.n; ++j) {
        switch (c.width[j]) {
            case 1: copy_kept<unsigned char>(c.in[j], c.out[j], row0, at, mine, lt, lane); break;
            case 2: copy_kept<unsigned short>(c.in[j], c.out[j], row0, at, mine, lt, lane); break;
            case 4: copy_kept<unsigned>(c.in[j], c.out[j], row0, at, mine, lt, lane); break;
            default: copy_kept<unsigned long long>(c.in[j], c.out[j], row0, at, mine, lt, lane); break;
        }
    }
}

// The closed range of a comparison with integer literals, in the column's type.
template <class W>
void int_range(const gx_predicate& q, W tmin, W tmax, pred_dev& p, int j) {
    const W a = (W)q.lo_i, b = (W)q.hi_i;
    W lo = tmin, hi = tmax;
    bool empty = false;
    switch (q.op) {
        case GX_CMP_LT: if (a <= tmin) empty = true; else hi = std::min<W>(tmax, a - 1); break;
        case GX_CMP_LE: if (a < tmin) empty = true; else hi = std::min(tmax, a); break;
        case GX_CMP_GT: if (a >= tmax) empty = true; else lo = std::max<W>(tmin, a + 1); break;
        case GX_CMP_GE: if (a > tmax) empty = true; else lo = std::max(tmin, a); break;
        case GX_CMP_EQ:
        case GX_CMP_NE: if (a < tmin || a > tmax) empty = true; else lo = hi = a; break;
        default:  // BETWEEN: a <= x < b
            if (b <= tmin || a > tmax || a >= b) empty = true;
            else { lo = std::max(tmin, a); hi = std::min<W>(tmax, b - 1); }
            break;
    }
    p.lo[j] = empty ? 1 : (uint64_t)lo;
    p.hi[j] = empty ? 0 : (uint64_t)hi;
}

void float_range(const gx_predicate& q, pred_dev& p, int j) {
    const double inf = std::numeric_limits<double>::infinity();
    double lo = -inf, hi = inf;
    bool empty = std::isnan(q.lo_f) || (q.op == GX_CMP_BETWEEN && std::isnan(q.hi_f));
    switch (q.op) {
        case GX_CMP_LT: empty |= q.lo_f == -inf; hi = std::nextafter(q.lo_f, -inf); break;
        case GX_CMP_LE: hi = q.lo_f; break;
        case GX_CMP_GT: empty |= q.lo_f == inf; lo = std::nextafter(q.lo_f, inf); break;
        case GX_CMP_GE: lo = q.lo_f; break;
        case GX_CMP_EQ:
        case GX_CMP_NE: lo = hi = q.lo_f; break;
        default: empty |= q.hi_f == -inf; lo = q.lo_f; hi = std::nextafter(q.hi_f, -inf); break;
    }
    if (empty) { lo = 1.0; hi = 0.0; }
    std::memcpy(&p.lo[j], &lo, 8);
    std::memcpy(&p.hi[j], &hi, 8);
}

void column_range(const gx_predicate& q, int type, pred_dev& p, int j) {
    p.negate[j] = q.op == GX_CMP_NE;
    p.type[j] = type;
    const int bits = 8 * size_of(type);
    if (is_float(type)) float_range(q, p, j);
    else if (is_signed_int(type)) int_range<int64_t>(q, INT64_MIN >> (64 - bits), INT64_MAX >> (64 - bits), p, j);
    else int_range<uint64_t>(q, 0, UINT64_MAX >> (64 - bits), p, j);
}

pred_dev make_preds(const gx_table_view* t, const gx_predicate* preds, int n, int combine) {
    require(t != nullptr, "select: null table");
    require(n >= 1 && n <= MAX_PRED, "select: 1 to " + std::to_string(MAX_PRED) + " predicates supported");
    require(preds != nullptr, "select: null predicates");
    require(combine == GX_COMBINE_AND || combine == GX_COMBINE_OR, "select: combine must be AND or OR");
    pred_dev p;
    std::memset(&p, 0, sizeof(p));
    p.n = n;
    p.combine = combine;
    for (int j = 0; j < n; ++j) {
        const gx_predicate& q = preds[j];
        require(q.column_index >= 0 && q.column_index < t->num_columns, "select: predicate column out of range");
        const gx_column_view& v = t->columns[q.column_index];
        require(is_numeric(v.type), "select: predicates on " + type_name(v.type) + " columns are not supported");
        require(q.op >= GX_CMP_LT && q.op <= GX_CMP_BETWEEN, "select: unknown comparison");
        col c = resolve(v);
        p.data[j] = c.data;
        column_range(q, v.type, p, j);
    }
    return p;
}

int64_t table_rows(const gx_table_view* t) {
    const int64_t n = t->num_columns ? t->columns[0].size : 0;
    for (int64_t c = 0; c < t->num_columns; ++c)
        require(t->columns[c].size == n, "select: columns differ in length");
    return n;
}

// Bits + scan + write of every column of `t` for the rows `p` keeps.  2^28 rows
// of a date and two 8-byte columns, BETWEEN keeping 40%: 1.72 ms a call
// (4.4 TB/s of the 28 bytes a row that the outputs need); 3.44 ms when the write
// kernel evaluated the predicate again and issued one load at a time.
void compact_rows(const gx_table_view* t, const pred_dev& p, int64_t n, cudaStream_t s, gx_table* out) {
    require(t->num_columns <= MAX_SEL_COLS, "select: at most " + std::to_string(MAX_SEL_COLS) + " columns");
    for (int64_t c = 0; c < t->num_columns; ++c)
        if (!is_numeric(t->columns[c].type)) fail(GX_EUNSUPPORTED, "compact: STRING columns are not supported");
    const int64_t ntiles = ceil_div(std::max<int64_t>(n, 1), SL_TILE);
    // Tile counts, their offsets, and one bit per row.
    const size_t bits_at = ((size_t)(2 * ntiles + 1) * 8 + 15) & ~size_t(15);
    dbuf tmp(bits_at + (size_t)ntiles * (SL_TILE / 8), s);
    int64_t* tc = tmp.get<int64_t>();
    int64_t* toff = tc + ntiles;
    unsigned* bits = reinterpret_cast<unsigned*>(tmp.get<char>() + bits_at);
    int64_t kept = 0;
    if (n > 0) {
        GX_PROF("select_count", s);
        k_sel_bits<<<(unsigned)ntiles, SL_NT, 0, s>>>(p, n, bits, tc);
        GX_LAUNCHED();
        exclusive_scan_i64(tc, toff, ntiles, s);
        kept = read_scalar(toff + ntiles, s);
    }
    sel_cols sc;
    std::memset(&sc, 0, sizeof(sc));
    out->cols.clear();
    for (int64_t c = 0; c < t->num_columns; ++c) {
        out->cols.push_back(make_col(t->columns[c].type, kept, s));
        col in = resolve(t->columns[c]);
        sc.in[sc.n] = in.data;
        sc.out[sc.n] = out->cols.back().buf.get();
        sc.width[sc.n] = size_of(in.type);
        ++sc.n;
    }
    if (kept > 0) {
        GX_PROF("select_write", s);
        k_sel_write<<<(unsigned)ntiles, SL_NT, 0, s>>>(bits, toff, sc);
        GX_LAUNCHED();
    }
    GX_CUDA(cudaStreamSynchronize(s));
}

}  // namespace

void select_to_bitmask(const gx_table_view* t, const gx_predicate* preds, int n, int combine, cudaStream_t s,
                       gx_column* mask) {
    pred_dev p = make_preds(t, preds, n, combine);
    const int64_t rows = table_rows(t);
    owned_col m = make_col(GX_BOOL8, rows, s);
    if (rows > 0) {
        k_sel_mask<<<(unsigned)ceil_div(rows, SL_TILE), SL_NT, 0, s>>>(p, rows, m.buf.get<uint8_t>());
        GX_LAUNCHED();
    }
    GX_CUDA(cudaStreamSynchronize(s));
    *mask = to_gx_column(std::move(m));
}

void select_rows(const gx_table_view* t, const gx_predicate* preds, int n, int combine, cudaStream_t s,
                 gx_table* out) {
    pred_dev p = make_preds(t, preds, n, combine);
    compact_rows(t, p, table_rows(t), s, out);
}

void compact_by_mask(const gx_table_view* t, const gx_column_view& mask, cudaStream_t s, gx_table* out) {
    require(t != nullptr, "compact: null table");
    require(size_of(mask.type) == 1, "compact: the mask must be a BOOL8 / 1-byte column");
    const int64_t n = table_rows(t);
    require(mask.size == n || t->num_columns == 0, "compact: mask length differs from the table's rows");
    pred_dev p;
    std::memset(&p, 0, sizeof(p));
    p.n = 1;
    p.data[0] = resolve(mask).data;
    gx_predicate q;
    std::memset(&q, 0, sizeof(q));
    q.op = GX_CMP_NE;
    column_range(q, GX_UINT8, p, 0);
    compact_rows(t, p, t->num_columns ? n : 0, s, out);
}

int64_t count_nonzero(const gx_column_view& v, cudaStream_t s) {
    col c = resolve(v);
    require(is_numeric(c.type), "count_nonzero: numeric column required");
    if (c.n == 0) return 0;
    gx_predicate q;
    std::memset(&q, 0, sizeof(q));
    q.column_index = 0;
    q.op = GX_CMP_NE;
    gx_table_view t{&v, 1};
    pred_dev p = make_preds(&t, &q, 1, GX_COMBINE_AND);
    const int64_t ntiles = ceil_div(c.n, SL_TILE);
    dbuf tc((size_t)ntiles * 8, s), toff((size_t)(ntiles + 1) * 8, s);
    k_sel_bits<<<(unsigned)ntiles, SL_NT, 0, s>>>(p, c.n, nullptr, tc.get<int64_t>());
    GX_LAUNCHED();
    exclusive_scan_i64(tc.get<int64_t>(), toff.get<int64_t>(), ntiles, s);
    return read_scalar(toff.get<int64_t>() + ntiles, s);
}

}  // namespace gx
