// WHERE programs evaluated for R rows of a thread at a time.
//
// eval_prog (common.cuh) interprets the postfix program row by row: every row
// re-decides each term's kind, column type and operator, which made the scans
// that used it issue-bound (two compares, one nullable column and four
// aggregates over 33M rows: 0.79 ms, 0.10 of the copy rate).  Here every term is decoded on the
// host, the decisions are uniform branches taken once per R rows, a term's
// outcome for the R rows is an R-bit mask, and the stack of outcomes is one
// 64-bit register (a program of at most 16 terms has at most 8 leaves).
#pragma once
#include <cstring>

#include "common.cuh"

namespace fdb {

enum : int32_t {
  kWhereF64 = 0,       // FLOAT64 column against a double
  kWhereI64,           // INT64 column against an int64
  kWhereI64AsF64,      // INT64 column widened to double (expr.rs:1122-1132)
  kWhereCode,          // UTF8 codes against a code; the NULL code fails
  kWhereCodeSet,
  kWhereNull,
  kWhereNotNull,
  kWhereAnd,
  kWhereOr
};

struct WhereTerm {
  int32_t kind;
  int32_t col;
  int32_t op;
  uint32_t set_len;    // CODE_SET: codes from here on never pass
  union {
    int64_t lit_i;
    double lit_f;
    const uint64_t* set;
  };
};

struct WhereProg {
  int32_t n;
  uint32_t nullable;   // bit c: column c has validity words
  // One comparison of an INT64 column with an int64 (where_one): the values
  // [one_lo, one_lo + one_span], or with one_not (all ones) those outside.
  uint32_t one_not;
  int64_t one_lo;
  uint64_t one_span;
  WhereTerm t[FDB_MAX_TERMS];
};

// x op lit over int64, as such a range.
inline void fill_where_range(WhereProg& w, int op, int64_t lit) {
  int64_t lo = INT64_MIN, hi = INT64_MAX;
  bool outside = false;
  switch (op) {
    case FDB_EQ: lo = hi = lit; break;
    case FDB_NE: lo = hi = lit; outside = true; break;
    case FDB_LE: hi = lit; break;
    case FDB_GT: hi = lit; outside = true; break;
    case FDB_GE: lo = lit; break;
    default: lo = lit; outside = true;  // <
  }
  w.one_lo = lo;
  w.one_span = (uint64_t)hi - (uint64_t)lo;
  w.one_not = outside ? 0xFFFFFFFFu : 0u;
}

// A checked program (fill_prog) over columns `cols`, decoded.
inline void fill_where(WhereProg& w, const PredProg& prog, const DevCol* cols, int ncols) {
  std::memset(&w, 0, sizeof(w));
  w.n = prog.n;
  for (int c = 0; c < ncols; ++c)
    if (cols[c].validity) w.nullable |= 1u << c;
  for (int i = 0; i < prog.n; ++i) {
    const fdb_pred_term& s = prog.t[i];
    WhereTerm& t = w.t[i];
    t.col = s.col;
    t.op = s.op;
    switch (s.kind) {
      case FDB_TERM_AND: t.kind = kWhereAnd; t.col = 0; break;
      case FDB_TERM_OR: t.kind = kWhereOr; t.col = 0; break;
      case FDB_TERM_IS_NULL: t.kind = kWhereNull; break;
      case FDB_TERM_IS_NOT_NULL: t.kind = kWhereNotNull; break;
      case FDB_TERM_CODE_SET:
        t.kind = kWhereCodeSet;
        t.set_len = s.lit_i <= 0 ? 0u : (s.lit_i >= (int64_t)kNullCode ? kNullCode : (uint32_t)s.lit_i);
        t.set = s.code_set;
        break;
      default:
        if (cols[s.col].dtype == FDB_FLOAT64) {
          t.kind = kWhereF64;
          t.lit_f = s.lit_type == FDB_FLOAT64 ? s.lit_f : (double)s.lit_i;
        } else if (cols[s.col].dtype == FDB_INT64) {
          t.kind = s.lit_type == FDB_FLOAT64 ? kWhereI64AsF64 : kWhereI64;
          if (s.lit_type == FDB_FLOAT64)
            t.lit_f = s.lit_f;
          else
            t.lit_i = s.lit_i;
        } else {
          t.kind = kWhereCode;
          t.lit_i = s.lit_i;
        }
    }
  }
  if (w.n == 1 && w.t[0].kind == kWhereI64) fill_where_range(w, w.t[0].op, w.t[0].lit_i);
}

// Programs that scans of NULL-free columns decide with less than where_mask: none,
// and one comparison of a numeric column (where_one).
enum WhereForm { kWhereNone, kWhereOne, kWhereAny };
inline WhereForm where_form(const WhereProg& w) {
  if (w.nullable || w.n > 1) return kWhereAny;
  if (w.n == 0) return kWhereNone;
  return w.t[0].kind <= kWhereI64AsF64 ? kWhereOne : kWhereAny;
}

// x[j] op lit for R values, the operator decided once (floating compares are
// IEEE ordered, != unordered, as cmp_op's).
template <int R, typename T>
__device__ __forceinline__ uint32_t cmp_mask(int op, const T (&x)[R], T lit) {
  uint32_t m = 0;
  switch (op) {
#define FDB_CMP_CASE(OP, SYM)                          \
  case OP:                                             \
    _Pragma("unroll") for (int j = 0; j < R; ++j) m |= (x[j] SYM lit ? 1u : 0u) << j; \
    break;
    FDB_CMP_CASE(FDB_EQ, ==)
    FDB_CMP_CASE(FDB_NE, !=)
    FDB_CMP_CASE(FDB_LT, <)
    FDB_CMP_CASE(FDB_LE, <=)
    FDB_CMP_CASE(FDB_GT, >)
    default:
#pragma unroll
      for (int j = 0; j < R; ++j) m |= (x[j] >= lit ? 1u : 0u) << j;
#undef FDB_CMP_CASE
  }
  return m;
}

// The rows i[j] of an accessor, `stride` (a multiple of 32) apart.
template <bool kFull, int R, typename T, class Acc>
__device__ __forceinline__ void where_load(T (&x)[R], const Acc& acc, int col, const uint32_t (&i)[R], uint32_t ok) {
#pragma unroll
  for (int j = 0; j < R; ++j) x[j] = (kFull || ((ok >> j) & 1u)) ? acc.template get<T>(col, i[j]) : T(0);
}

// Validity bits of rows i[j].  The rows are a multiple of 32 apart, so one
// word address and one shift serve them all: the loads differ by constants.
template <bool kFull, int R, int kStride, class Acc>
__device__ __forceinline__ uint32_t valid_mask(const DevCol& c, const Acc& acc, const uint32_t (&i)[R], uint32_t ok) {
  static_assert(kStride % 32 == 0, "rows of a thread are whole validity words apart");
  const uint64_t b = c.voff + acc.row(i[0]);
  const uint32_t* w = reinterpret_cast<const uint32_t*>(c.validity) + (b >> 5);
  const int sh = (int)(b & 31);
  uint32_t m = 0;
#pragma unroll
  for (int j = 0; j < R; ++j)
    if (kFull || ((ok >> j) & 1u)) m |= ((__ldg(w + j * (kStride / 32)) >> sh) & 1u) << j;
  return m;
}

// Brings the validity words of rows [row0, row0 + rows) of every nullable
// column into L2 (128 bytes hold 1024 rows).
__device__ __forceinline__ void prefetch_valid(uint32_t nullable, const DevCol* cols, uint64_t row0, uint32_t rows) {
  for (int c = 0; nullable >> c; ++c) {
    if (!((nullable >> c) & 1u)) continue;
    const uint64_t b0 = (cols[c].voff + row0) >> 3, b1 = (cols[c].voff + row0 + rows - 1) >> 3;
    const unsigned char* base = reinterpret_cast<const unsigned char*>(cols[c].validity);
    for (uint64_t b = b0 & ~127ull; b <= b1; b += 128)
      asm volatile("prefetch.global.L2 [%0];" ::"l"(base + (b < b0 ? b0 : b)));
  }
}

// Validity of every nullable column: R bits per column, column c from bit c*R.
template <bool kFull, int R, int kStride, class Acc>
__device__ __forceinline__ uint32_t valid_masks(uint32_t nullable, const DevCol* cols, const Acc& acc,
                                                const uint32_t (&i)[R], uint32_t ok) {
  static_assert(4 * R <= 32, "four columns' masks in one word");
  uint32_t v = 0xFFFFFFFFu;
  if (nullable) {
#pragma unroll
    for (int c = 0; c < 4; ++c)
      if ((nullable >> c) & 1u)
        v &= ~(((1u << R) - 1u) << (c * R)) | (valid_mask<kFull, R, kStride>(cols[c], acc, i, ok) << (c * R));
  }
  return v;
}

// The rows of i[j] (those set in `ok`) that pass; `valid` from valid_masks.
template <bool kFull, int R, class Acc>
__device__ __forceinline__ uint32_t where_mask(const WhereProg& w, const Acc& acc, const DevCol* cols,
                                               const uint32_t (&i)[R], uint32_t ok, uint32_t valid) {
  static_assert(R <= 8, "eight R-bit outcomes in 64 bits");
  constexpr uint32_t kAll = R == 32 ? 0xFFFFFFFFu : (1u << R) - 1u;
  if (w.n == 0) return ok;
  uint64_t below = 0;  // outcomes under the top one
  uint32_t top = 0;
  for (int k = 0; k < w.n; ++k) {
    const WhereTerm& t = w.t[k];
    if (t.kind >= kWhereAnd) {
      const uint32_t b = (uint32_t)below & kAll;
      below >>= R;
      top = t.kind == kWhereAnd ? (top & b) : (top | b);
      continue;
    }
    below = (below << R) | top;
    const uint32_t v = (valid >> (t.col * R)) & kAll;
    switch (t.kind) {
      case kWhereF64: {
        double x[R];
        where_load<kFull, R>(x, acc, t.col, i, ok);
        top = cmp_mask<R, double>(t.op, x, t.lit_f) & v;
        break;
      }
      case kWhereI64: {
        int64_t x[R];
        where_load<kFull, R>(x, acc, t.col, i, ok);
        top = cmp_mask<R, int64_t>(t.op, x, t.lit_i) & v;
        break;
      }
      case kWhereI64AsF64: {
        int64_t y[R];
        double x[R];
        where_load<kFull, R>(y, acc, t.col, i, ok);
#pragma unroll
        for (int j = 0; j < R; ++j) x[j] = (double)y[j];
        top = cmp_mask<R, double>(t.op, x, t.lit_f) & v;
        break;
      }
      default: {
        // IS [NOT] NULL of a numeric column is its validity; the others read
        // the codes (a UTF8 cell is NULL through its validity or its code).
        uint32_t null = ~v & kAll;
        if (cols[t.col].dtype == FDB_UTF8) {
          uint32_t x[R];
          where_load<kFull, R>(x, acc, t.col, i, ok);
#pragma unroll
          for (int j = 0; j < R; ++j) null |= (x[j] == kNullCode ? 1u : 0u) << j;
          if (t.kind == kWhereCode) {
            int64_t y[R];
#pragma unroll
            for (int j = 0; j < R; ++j) y[j] = (int64_t)x[j];
            top = cmp_mask<R, int64_t>(t.op, y, t.lit_i);
          } else if (t.kind == kWhereCodeSet) {
            top = 0;
#pragma unroll
            for (int j = 0; j < R; ++j)
              if (x[j] < t.set_len) top |= (uint32_t)((__ldg(t.set + (x[j] >> 6)) >> (x[j] & 63)) & 1ull) << j;
          }
        } else if (t.kind == kWhereCodeSet) {
          top = 0;
#pragma unroll
          for (int j = 0; j < R; ++j) top |= (0u < t.set_len && (__ldg(t.set) & 1ull) ? 1u : 0u) << j;
        }
        if (t.kind == kWhereNull)
          top = null;
        else if (t.kind == kWhereNotNull)
          top = ~null & kAll;
        else
          top &= ~null;
      }
    }
  }
  return kFull ? top : (top & ok);
}

// where_mask for one comparison (kWhereOne), which is the program's first term: its
// fields are read at fixed places of the parameters.
template <bool kFull, int R, class Acc>
__device__ __forceinline__ uint32_t where_one(const WhereProg& w, const Acc& acc, const uint32_t (&i)[R],
                                              uint32_t ok) {
  const WhereTerm& t = w.t[0];
  uint32_t m = 0;
  if (t.kind == kWhereF64) {
    double x[R];
    where_load<kFull, R>(x, acc, t.col, i, ok);
    m = cmp_mask<R, double>(t.op, x, t.lit_f);
  } else {
    int64_t y[R];
    where_load<kFull, R>(y, acc, t.col, i, ok);
    if (t.kind == kWhereI64) {
      const uint64_t lo = (uint64_t)w.one_lo, span = w.one_span;
#pragma unroll
      for (int j = 0; j < R; ++j) m |= ((uint64_t)y[j] - lo <= span ? 1u : 0u) << j;
      m = (m ^ w.one_not) & ((1u << R) - 1u);
    } else {
      double x[R];
#pragma unroll
      for (int j = 0; j < R; ++j) x[j] = (double)y[j];
      m = cmp_mask<R, double>(t.op, x, t.lit_f);
    }
  }
  return kFull ? m : (m & ok);
}

}  // namespace fdb
