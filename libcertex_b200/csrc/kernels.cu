// Plain CUDA kernels of the exact search path: per-row init values of the integer screen, the per-query threshold,
// exact fp64 verification with top-k selection, the dense (unscreened) path, output conversion and the merge of
// per-shard answers.
//
// The exact score of a pair follows `warp_score` / `exact_score` of the reference
// (cpp/src/neighbors/certex/detail/certex_kernels.cuh:247-273, cpp/tests/neighbors/ann_certex.cuh:78-99):
//   L2 sum (q-x)^2, inner product |q|^2 - 2<q,x>, cosine 2 - 2<q,x>/sqrt(max(|q|^2 |x|^2, 1e-300)).
// Each thread walks one stored row from coordinate 0 to d-1 and rounds every product and every sum on its own
// (__dmul_rn / __dadd_rn, never a fused multiply-add), which is the order and rounding of the sequential CPU loop: the
// fp64 scores are bit-identical to it for every element type. Rows are read with 16-byte loads.
//
// The order among equal scores is (score, id) everywhere (selection, sort, merge).
#include "kernels.cuh"

#include "screen_i8.cuh"  // kNeverInit

#include <cub/cub.cuh>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <math_constants.h>

#include <algorithm>
#include <type_traits>

namespace certex_b200 {

namespace {

// ------------------------------------------------------------------------------------------- element access
template <typename T>
struct Elems;
// The double of a FINITE float32 (bits f) without the conversion instruction, whose pipe does about two per clock and
// SM: the float's sign, exponent field and mantissa are placed in a double's fields as they are, which gives
// x * 2^-896 (a subnormal float lands on a subnormal double, zero on zero), and one multiplication by 2^896 - exact,
// a power of two - restores x. Infinities and NaNs would come out finite: callers use it only on stored rows that
// passed the fp16 range check of the screen.
__device__ __forceinline__ double widen_finite(uint32_t f)
{
  const uint32_t hi = ((f & 0x7fffffffu) >> 3) | (f & 0x80000000u);
  return __dmul_rn(__hiloint2double(static_cast<int>(hi), static_cast<int>(f << 29)), 0x1p896);
}

template <>
struct Elems<float> {
  static constexpr int kPerVec = 4;
  __device__ static void unpack(const uint4& w, double (&o)[4])
  {
    o[0] = double(__uint_as_float(w.x)), o[1] = double(__uint_as_float(w.y));
    o[2] = double(__uint_as_float(w.z)), o[3] = double(__uint_as_float(w.w));
  }
  __device__ static void unpack_finite(const uint4& w, double (&o)[4])
  {
    o[0] = widen_finite(w.x), o[1] = widen_finite(w.y), o[2] = widen_finite(w.z), o[3] = widen_finite(w.w);
  }
  __device__ static double one(const void* p, int64_t i) { return double(static_cast<const float*>(p)[i]); }
};
template <>
struct Elems<__half> {
  static constexpr int kPerVec = 8;
  __device__ static void unpack(const uint4& w, double (&o)[8])
  {
    const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const __half2 h = *reinterpret_cast<const __half2*>(&u[i]);
      o[2 * i]        = double(__low2float(h));
      o[2 * i + 1]    = double(__high2float(h));
    }
  }
  __device__ static void unpack_finite(const uint4& w, double (&o)[8])
  {
    const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const __half2 h = *reinterpret_cast<const __half2*>(&u[i]);
      o[2 * i]        = widen_finite(__float_as_uint(__low2float(h)));
      o[2 * i + 1]    = widen_finite(__float_as_uint(__high2float(h)));
    }
  }
  __device__ static double one(const void* p, int64_t i) { return double(__half2float(static_cast<const __half*>(p)[i])); }
};
template <>
struct Elems<int8_t> {
  static constexpr int kPerVec = 16;
  __device__ static void unpack(const uint4& w, double (&o)[16])
  {
    const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int i = 0; i < 16; ++i) { o[i] = double(int(int8_t((u[i >> 2] >> (8 * (i & 3))) & 0xffu))); }
  }
  __device__ static double one(const void* p, int64_t i) { return double(static_cast<const int8_t*>(p)[i]); }
};
template <>
struct Elems<uint8_t> {
  static constexpr int kPerVec = 16;
  __device__ static void unpack(const uint4& w, double (&o)[16])
  {
    const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int i = 0; i < 16; ++i) { o[i] = double(int((u[i >> 2] >> (8 * (i & 3))) & 0xffu)); }
  }
  __device__ static double one(const void* p, int64_t i) { return double(static_cast<const uint8_t*>(p)[i]); }
};

__device__ __forceinline__ bool admitted(const Admit& a, int64_t q, int64_t row)
{
  if (a.removed && a.removed[row]) { return false; }
  if (a.bits) {
    const int64_t bit = a.bitmap_cols > 0 ? q * a.bitmap_cols + row : row;
    if (((a.bits[bit >> 5] >> (bit & 31)) & 1u) == 0u) { return false; }
  }
  if (a.row_labels) {
    const int32_t l = a.row_labels[row];
    if (l < 0 || l != a.query_labels[q]) { return false; }
  }
  return true;
}

// Accumulators of NQ queries against one stored row, coordinates in order. STORED_XX (cosine): |x|^2 is not summed here,
// the caller sets xx from the value kept with the row (the same sum, made once when the row was added).
template <int METRIC, int NQ, bool STORED_XX = false>
struct Acc {
  double s[NQ];  // L2: sum of squared differences; otherwise: inner product
  double xx;
  __device__ void clear()
  {
#pragma unroll
    for (int b = 0; b < NQ; ++b) { s[b] = 0; }
    xx = 0;
  }
  // qd: queries as doubles in shared memory, query b at qd + b * ldq
  __device__ __forceinline__ void add(double x, const double* qd, int ldq, int t)
  {
#pragma unroll
    for (int b = 0; b < NQ; ++b) {
      const double a = qd[b * ldq + t];
      if constexpr (METRIC == kL2) {
        const double diff = __dsub_rn(a, x);
        s[b]              = __dadd_rn(s[b], __dmul_rn(diff, diff));
      } else {
        s[b] = __dadd_rn(s[b], __dmul_rn(a, x));
      }
    }
    if constexpr (METRIC == kCos && !STORED_XX) { xx = __dadd_rn(xx, __dmul_rn(x, x)); }
  }
  // the same for one query whose coordinate the caller has loaded (a)
  __device__ __forceinline__ void add1(double x, double a)
  {
    if constexpr (METRIC == kL2) {
      const double diff = __dsub_rn(a, x);
      s[0]              = __dadd_rn(s[0], __dmul_rn(diff, diff));
    } else {
      s[0] = __dadd_rn(s[0], __dmul_rn(a, x));
    }
    if constexpr (METRIC == kCos && !STORED_XX) { xx = __dadd_rn(xx, __dmul_rn(x, x)); }
  }
  __device__ __forceinline__ double result(int b, double qq) const
  {
    if constexpr (METRIC == kL2) {
      return s[b];
    } else if constexpr (METRIC == kIP) {
      return __dsub_rn(qq, __dmul_rn(2.0, s[b]));
    } else {
      const double den = fmax(__dmul_rn(qq, xx), 1e-300);
      return __dsub_rn(2.0, __ddiv_rn(__dmul_rn(2.0, s[b]), __dsqrt_rn(den)));
    }
  }
};

// Walks one stored row (16-byte loads) and feeds every coordinate to `acc`. FINITE: the row holds no infinity or NaN
// (float types; see widen_finite).
template <typename T, int METRIC, int NQ, bool FINITE = false>
__device__ __forceinline__ void scan_row(const uint8_t* row, int d, const double* qd, int ldq, Acc<METRIC, NQ>& acc)
{
  constexpr int V   = Elems<T>::kPerVec;
  const uint4* p    = reinterpret_cast<const uint4*>(row);
  const int n_full  = d / V;
  for (int c = 0; c < n_full; ++c) {
    const uint4 w = __ldg(p + c);
    double x[V];
    if constexpr (FINITE) {
      Elems<T>::unpack_finite(w, x);
    } else {
      Elems<T>::unpack(w, x);
    }
#pragma unroll
    for (int e = 0; e < V; ++e) { acc.add(x[e], qd, ldq, c * V + e); }
  }
  for (int t = n_full * V; t < d; ++t) { acc.add(Elems<T>::one(row, t), qd, ldq, t); }
}

// Queries as doubles into shared memory and |q|^2 summed in coordinate order by one thread per query.
template <typename T>
__device__ void load_queries(const void* queries, size_t qpitch, const int64_t* qidx, int nqb, int d, double* qd, int ldq, double* qq)
{
  for (int b = 0; b < nqb; ++b) {
    const uint8_t* src = static_cast<const uint8_t*>(queries) + static_cast<size_t>(qidx[b]) * qpitch;
    for (int t = threadIdx.x; t < d; t += blockDim.x) { qd[b * ldq + t] = Elems<T>::one(src, t); }
  }
  __syncthreads();
  if (threadIdx.x < nqb) {
    double a = 0;
    for (int t = 0; t < d; ++t) {
      const double v = qd[threadIdx.x * ldq + t];
      a              = __dadd_rn(a, __dmul_rn(v, v));
    }
    qq[threadIdx.x] = a;
  }
  __syncthreads();
}

// ------------------------------------------------------------------------------------------- sorting helpers
__device__ __forceinline__ bool pair_less(double sa, int64_t ia, double sb, int64_t ib)
{
  return sa < sb || (sa == sb && ia < ib);
}

// In-place bitonic sort of n2 (a power of two) (score, id) pairs in shared memory, ascending by (score, id).
template <typename IdT>
__device__ void bitonic_sort(double* s, IdT* id, int n2)
{
  for (int size = 2; size <= n2; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      __syncthreads();
      for (int i = threadIdx.x; i < (n2 >> 1); i += blockDim.x) {
        const int lo   = 2 * i - (i & (stride - 1));
        const int hi   = lo + stride;
        const bool asc = (lo & size) == 0;
        const double a = s[lo], b = s[hi];
        const IdT ia = id[lo], ib = id[hi];
        const bool swap = asc ? pair_less(b, ib, a, ia) : pair_less(a, ia, b, ib);
        if (swap) {
          s[lo] = b, s[hi] = a;
          id[lo] = ib, id[hi] = ia;
        }
      }
    }
  }
  __syncthreads();
}

// In-place bitonic sort of n2 (a power of two) 64-bit keys in shared memory, ascending.
__device__ void bitonic_sort_keys(unsigned long long* key, int n2)
{
  for (int size = 2; size <= n2; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      __syncthreads();
      for (int i = threadIdx.x; i < (n2 >> 1); i += blockDim.x) {
        const int lo                 = 2 * i - (i & (stride - 1));
        const int hi                 = lo + stride;
        const unsigned long long a   = key[lo], b = key[hi];
        const bool asc               = (lo & size) == 0;
        if (asc ? b < a : a < b) { key[lo] = b, key[hi] = a; }
      }
    }
  }
  __syncthreads();
}

__device__ __forceinline__ unsigned long long ordered_key(double v)
{
  const unsigned long long b = static_cast<unsigned long long>(__double_as_longlong(v));
  return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}

__host__ __device__ inline int next_pow2(int v)
{
  int p = 1;
  while (p < v) { p <<= 1; }
  return p;
}

// ------------------------------------------------------------------------------------------- build-side kernels
// Eight lanes per row, 16 bytes per lane and step.
template <typename T>
__global__ void row_init_kernel(const uint8_t* vectors, size_t pitch, int d, int metric, const uint8_t* removed,
                                int64_t row0, int64_t n, int64_t n_pad, int32_t* init)
{
  const int64_t gt  = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int64_t r   = row0 + (gt >> 3);
  const int sub     = threadIdx.x & 7;
  const bool in     = r < row0 + n;
  long long sum     = 0;
  if (in && metric == kL2) {
    const uint4* p  = reinterpret_cast<const uint4*>(vectors + static_cast<size_t>(r) * pitch);
    const int n_vec = (d + 15) / 16;  // rows are zero padded to the pitch
    for (int c = sub; c < n_vec; c += 8) {
      const uint4 w       = __ldg(p + c);
      const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const uint32_t byte = (u[i >> 2] >> (8 * (i & 3))) & 0xffu;
        const int v         = sizeof(T) == 1 && T(-1) < T(0) ? int(int8_t(byte)) : int(byte);
        sum += v * v;
      }
    }
  }
  sum += __shfl_xor_sync(0xffffffffu, sum, 1);
  sum += __shfl_xor_sync(0xffffffffu, sum, 2);
  sum += __shfl_xor_sync(0xffffffffu, sum, 4);
  if (sub == 0 && r < n_pad) {
    int32_t v = kNeverInit;
    if (in && !(removed && removed[r])) { v = metric == kL2 ? -static_cast<int32_t>(sum >> 1) : 0; }
    init[r] = v;
  }
}

// e of the anchors in tile order: out[t * 256 + c] = init[(c * n_tiles + t) * stride].
// With a bitset (one bit per id, set = keep) the anchors the filter drops get `never`, like removed rows: the threshold
// then comes from anchors the search may return.
__global__ void gather_init_kernel(const int32_t* init, int64_t stride, int64_t n_tiles, int32_t* out, const uint32_t* bits,
                                   const int32_t* perm, int32_t never)
{
  const int64_t j = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (j < n_tiles * kBaseTile) {
    const int64_t t = j / kBaseTile, c = j % kBaseTile;
    const int64_t r = (c * n_tiles + t) * stride;
    int32_t e       = init[r];
    if (bits) {
      const int32_t id = perm[r];
      if (((bits[id >> 5] >> (id & 31)) & 1u) == 0u) { e = never; }
    }
    out[j] = e;
  }
}

// Smallest e of every chain of 16 columns in the tile order of the chained anchor pass:
// out[t * 16 + i] = min over w < 16 of init[t * stride_t + i * stride_i + w * stride_w]  (int32 values, or floats by their bits).
__global__ void gather_chain_min_kernel(const int32_t* init, int64_t stride_w, int64_t stride_i, int64_t stride_t,
                                        int64_t n_tiles, int32_t* out, int is_float)
{
  const int64_t j = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (j >= n_tiles * (kBaseTile / kChainRows)) { return; }
  const int64_t t = j / (kBaseTile / kChainRows), i = j % (kBaseTile / kChainRows);
  const int32_t* src = init + t * stride_t + i * stride_i;
  if (is_float) {
    float m = __int_as_float(src[0]);
    for (int w = 1; w < kChainRows; ++w) { m = fminf(m, __int_as_float(src[w * stride_w])); }
    out[j] = __float_as_int(m);
  } else {
    int32_t m = src[0];
    for (int w = 1; w < kChainRows; ++w) { m = min(m, src[w * stride_w]); }
    out[j] = m;
  }
}

__global__ void remove_kernel(const int64_t* ids, int64_t n_ids, int64_t size, uint8_t* removed, int32_t* init,
                              const int32_t* inv, unsigned long long* n_new, int32_t never)
{
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n_ids) { return; }
  const int64_t id = ids[i];
  if (id < 0 || id >= size) { return; }
  // byte-wide exchange through the containing 32-bit word
  uint32_t* word       = reinterpret_cast<uint32_t*>(removed + (id & ~int64_t(3)));
  const uint32_t bit   = 1u << (8 * (id & 3));
  const uint32_t prev  = atomicOr(word, bit);
  if ((prev & bit) == 0u) { atomicAdd(n_new, 1ull); }
  if (init) { init[inv ? inv[id] : id] = never; }
}

// cmax[c] = max of e over rows [16c, 16c + 16) for chains c0 .. c0 + n - 1 (e padded with kNeverInit).
__global__ void chain_max_kernel(const int32_t* init, int64_t c0, int64_t n, int32_t* cmax)
{
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) { return; }
  const int4* e = reinterpret_cast<const int4*>(init + (c0 + i) * 16);
  int m         = kNeverInit;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int4 t = e[k];
    m            = max(max(max(m, t.x), max(t.y, t.z)), t.w);
  }
  cmax[c0 + i] = m;
}

// The chains that hold removed ids get their maximum recomputed (after remove_kernel has marked the rows).
__global__ void chain_max_of_ids_kernel(const int64_t* ids, int64_t n_ids, int64_t size, const int32_t* inv,
                                        const int32_t* init, int32_t* cmax, int is_float)
{
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n_ids) { return; }
  const int64_t id = ids[i];
  if (id < 0 || id >= size) { return; }
  const int64_t c = (inv ? inv[id] : id) / 16;
  if (is_float) {
    float m = -CUDART_INF_F;
    for (int k = 0; k < 16; ++k) { m = fmaxf(m, __int_as_float(init[c * 16 + k])); }
    cmax[c] = __float_as_int(m);
  } else {
    int m = kNeverInit;
    for (int k = 0; k < 16; ++k) { m = max(m, init[c * 16 + k]); }
    cmax[c] = m;
  }
}

// keys[j] = -e[j] (half the squared norm, ascending sort key; for floats the bits of the non-negative float),
// vals[j] = id0 + j.
__global__ void sort_keys_kernel(const int32_t* e, int64_t n, int32_t id0, uint32_t* keys, int32_t* vals, int is_float)
{
  const int64_t j = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (j < n) {
    keys[j] = is_float ? __float_as_uint(-__int_as_float(e[j])) : static_cast<uint32_t>(-e[j]);
    vals[j] = id0 + static_cast<int32_t>(j);
  }
}

// Sorted batch -> index arrays: perm[row0 + j] = id, inv[id] = row0 + j, init[row0 + j] = -key, and the code row.
// `src` holds the code row of id at src + (id - src_id0) * pitch.
__global__ void place_sorted_kernel(const uint32_t* keys, const int32_t* ids, int64_t n, int64_t row0, const uint8_t* src,
                                    int64_t src_id0, size_t pitch, uint8_t* codes, int32_t* perm, int32_t* inv, int32_t* init,
                                    int metric, int is_float)
{
  const int64_t gt   = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int chunks   = static_cast<int>(pitch / 16);
  const int64_t j    = gt / chunks;
  const int c        = static_cast<int>(gt % chunks);
  if (j >= n) { return; }
  const int32_t id = ids[j];
  reinterpret_cast<uint4*>(codes + static_cast<size_t>(row0 + j) * pitch)[c] =
    __ldg(reinterpret_cast<const uint4*>(src + static_cast<size_t>(id - src_id0) * pitch) + c);
  if (c == 0) {
    perm[row0 + j] = id;
    inv[id]        = static_cast<int32_t>(row0 + j);
    init[row0 + j] = metric != kL2 ? 0 : is_float ? __float_as_int(-__uint_as_float(keys[j])) : -static_cast<int32_t>(keys[j]);
  }
}

__global__ void mask_removed_kernel(int32_t* e, const uint8_t* removed, int64_t n, int32_t never)
{
  const int64_t j = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (j < n && removed[j]) { e[j] = never; }
}

__global__ void fill_i32_kernel(int32_t* p, int64_t n, int32_t v)
{
  const int64_t j = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (j < n) { p[j] = v; }
}

// ------------------------------------------------------------------------------------------- fp16 codes of float data
// G lanes per row: the row rounded to fp16 (for the cosine metric: the row scaled to unit length first), and what the
// certified threshold test needs to know about the rounding:
//   |h|           norm of the fp16 code                          (rounded up)
//   |y - h|       norm of the rounding residual                  (rounded up)
//   e = -|x|^2/2  per-row term of the L2 value <q, x> - |x|^2/2  (rounded up; 0 for inner product and cosine)
// All sums are fp64. maxima[0..2] collect the largest |h|, |y - h| and |e| as float bits (non-negative floats order
// like their bits); maxima[3] is raised when a coordinate does not fit fp16.
//
// Bound by memory (the row in, its code out). The blocks are few enough to walk the rows in a grid stride of many turns, and a lane keeps the largest squared norms it has seen (a norm rounds up monotonically in its square), so that
// a block touches the three counters once: an atomic per row on the same three words held the whole pass at their rate
// (262 144 rows of 128 halves: 534 us, 0.25 TB/s; now 43 us, 3.1 TB/s). 16-byte loads; a row is split over 8 lanes when that leaves a lane at
// most four of them, so that short rows do not leave most of a warp without a coordinate, else over the whole warp.
constexpr int kEncodeThreads = 256;
// Two turns of the blocks that an SM holds (4 of 58 registers a thread for halves, 5 of 48 for floats). Us at 4 / 5 / 8 / 10 blocks
// an SM: 262 144 x 128 halves 44 / 55 / 44 / 46, 1 M x 768 halves 858 / 1042 / 850 / 877, 1 M x 768 floats (cosine) 1083 / 1039 /
// 1026 / 1005, 1 M x 128 floats 199 / 181 / 201 / 180.
constexpr int kEncodeBlocks  = 148 * 8;
template <typename T, int G>
__global__ void __launch_bounds__(kEncodeThreads) encode_f16_rows_kernel(const uint8_t* vectors, size_t pitch, int d, int metric,
                                                                         int64_t n, uint8_t* codes, size_t code_pitch, float* e,
                                                                         unsigned int* maxima)
{
  constexpr int V      = Elems<T>::kPerVec;
  constexpr int kRows  = kEncodeThreads / G;  // rows a block works on at a time
  const int sub        = threadIdx.x % G;
  const int n_vec      = (d + V - 1) / V;     // rows are zero padded to 16 bytes
  const int d_pad      = static_cast<int>(code_pitch / 2);
  const int64_t stride = static_cast<int64_t>(gridDim.x) * kRows;
  double hh_max = 0, rr_max = 0;
  float e_max   = 0;
  bool bad      = false;
  // the same number of turns for every lane of a warp: the sums of a row cross lanes
  for (int64_t row0 = static_cast<int64_t>(blockIdx.x) * kRows; row0 < n; row0 += stride) {
    const int64_t row  = row0 + threadIdx.x / G;
    const bool in      = row < n;
    const uint4* src   = reinterpret_cast<const uint4*>(vectors + static_cast<size_t>(in ? row : 0) * pitch);
    __half* dst        = reinterpret_cast<__half*>(codes + static_cast<size_t>(in ? row : 0) * code_pitch);
    double xx = 0, hh = 0, rr = 0, scale = 1.0;
    if (metric == kCos) {
      for (int c = sub; in && c < n_vec; c += G) {
        double x[V];
        Elems<T>::unpack(__ldg(src + c), x);
#pragma unroll
        for (int i = 0; i < V; ++i) { xx += x[i] * x[i]; }
      }
#pragma unroll
      for (int o = G / 2; o > 0; o >>= 1) { xx += __shfl_xor_sync(0xffffffffu, xx, o); }
      scale = xx > 0 ? 1.0 / sqrt(xx) : 0.0;
    }
    for (int c = sub; in && c < n_vec; c += G) {
      double x[V];
      Elems<T>::unpack(__ldg(src + c), x);
      __align__(16) __half h[V];
#pragma unroll
      for (int i = 0; i < V; ++i) {
        if (metric != kCos) { xx += x[i] * x[i]; }
        const double y  = x[i] * scale;
        h[i]            = __double2half(y);
        const double hf = static_cast<double>(__half2float(h[i]));
        bad |= isinf(hf) || isnan(hf);
        hh += hf * hf;
        rr += (y - hf) * (y - hf);
      }
      if constexpr (V == 8) {
        reinterpret_cast<uint4*>(dst)[c] = *reinterpret_cast<const uint4*>(h);
      } else {
        reinterpret_cast<uint2*>(dst)[c] = *reinterpret_cast<const uint2*>(h);
      }
    }
    for (int t = n_vec * V + sub; in && t < d_pad; t += G) { dst[t] = __float2half_rn(0.f); }
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) {
      if (metric != kCos) { xx += __shfl_xor_sync(0xffffffffu, xx, o); }
      hh += __shfl_xor_sync(0xffffffffu, hh, o);
      rr += __shfl_xor_sync(0xffffffffu, rr, o);
    }
    if (in) {
      // a sum that is not a number (a coordinate was not finite: `bad`) must not end up below the others
      hh_max = hh > hh_max || isnan(hh) ? hh : hh_max;
      rr_max = rr > rr_max || isnan(rr) ? rr : rr_max;
      const float ev = metric == kL2 ? __double2float_ru(-0.5 * xx) : 0.f;
      e_max          = fmaxf(e_max, fabsf(ev));
      if (sub == 0) { e[row] = ev; }
    }
  }
  // the unit-length scaling is itself rounded (fp64): a relative 2^-50 on every coordinate, far inside the slack
  uint32_t n1 = __float_as_uint(__double2float_ru(sqrt(hh_max) * (1.0 + 1e-9)));
  uint32_t n2 = __float_as_uint(__double2float_ru(sqrt(rr_max) * (1.0 + 1e-9) + (metric == kCos ? 1e-12 : 0.0)));
  uint32_t em = __float_as_uint(e_max);
  n1 = __reduce_max_sync(0xffffffffu, n1);
  n2 = __reduce_max_sync(0xffffffffu, n2);
  em = __reduce_max_sync(0xffffffffu, em);
  __shared__ uint32_t s_max[3][kEncodeThreads / 32];
  if ((threadIdx.x & 31) == 0) {
    const int w = threadIdx.x >> 5;
    s_max[0][w] = n1, s_max[1][w] = n2, s_max[2][w] = em;
  }
  const int any_bad = __syncthreads_or(bad);
  if (threadIdx.x < 3) {
    uint32_t m = 0;
    for (int w = 0; w < kEncodeThreads / 32; ++w) { m = max(m, s_max[threadIdx.x][w]); }
    atomicMax(maxima + threadIdx.x, m);
  }
  if (threadIdx.x == 0 && any_bad) { atomicExch(maxima + 3, 1u); }
}

// One warp per query: the fp16 code of the query and shift[q] = 2 (E + slack), the amount by which the k-th largest
// group maximum of the anchors is lowered to become the screen's threshold. With h = fp16(q), x~ = fp16 code of a row:
//   <q, x> = <h, x~> + <q - h, x~> + <q, x - x~>,   |<q - h, x~>| <= |q - h| |x~|,   |<q, x - x~>| <= |q| |x - x~|
//   |acc - <h, x~>| <= gamma |h| |x~|    (fp32 accumulation of exact fp16 products, gamma = (d + 16) 2^-20)
// so |acc - <q, x>| <= E(q) = (|q - h| + gamma |h|) N1 + |q| N2 with N1, N2 the largest |x~|, |x - x~| of the index.
// slack covers the fp32 additions of the epilogue, the rounding of e and of the exact fp64 scores: 2^-18 (|h| N1 + Emax).
// The anchors give a value every one of k rows certainly reaches (their group maximum minus E + slack); a row is
// kept unless its value certainly lies below that (its maximum plus E + slack): hence twice.
template <typename T>
__global__ void encode_f16_queries_kernel(const uint8_t* queries, size_t qpitch, int d, int64_t nq, int64_t nq_pad, uint8_t* codes,
                                          size_t code_pitch, float n1max, float n2max, float emax, float* shift,
                                          unsigned int* overflow)
{
  const int64_t row = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int lane    = threadIdx.x & 31;
  if (row >= nq_pad) { return; }
  const uint8_t* src = queries + static_cast<size_t>(row) * qpitch;
  __half* dst        = reinterpret_cast<__half*>(codes + static_cast<size_t>(row) * code_pitch);
  const int d_pad    = static_cast<int>(code_pitch / 2);
  if (row >= nq) {  // rows that fill the last query tile
    for (int t = lane; t < d_pad; t += 32) { dst[t] = __float2half_rn(0.f); }
    return;
  }
  double qq = 0, hh = 0, rr = 0;
  bool bad = false;
  for (int t = lane; t < d_pad; t += 32) {
    __half h = __float2half_rn(0.f);
    if (t < d) {
      const double y  = Elems<T>::one(src, t);
      h               = __double2half(y);
      const double hf = static_cast<double>(__half2float(h));
      bad |= isinf(hf) || isnan(hf);
      qq += y * y;
      hh += hf * hf;
      rr += (y - hf) * (y - hf);
    }
    dst[t] = h;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    qq += __shfl_xor_sync(0xffffffffu, qq, o);
    hh += __shfl_xor_sync(0xffffffffu, hh, o);
    rr += __shfl_xor_sync(0xffffffffu, rr, o);
  }
  bad = __any_sync(0xffffffffu, bad);
  if (lane == 0) {
    const double gamma = (d + 16) * 9.5367431640625e-07;  // 2^-20
    const double nqh = sqrt(hh) * (1.0 + 1e-9), dq = sqrt(rr) * (1.0 + 1e-9), nqn = sqrt(qq) * (1.0 + 1e-9);
    const double E     = (dq + gamma * nqh) * n1max + nqn * n2max;
    const double slack = 3.814697265625e-06 * (nqh * n1max + emax);  // 2^-18
    shift[row]         = __double2float_ru(2.0 * (E + slack) * (1.0 + 1e-6));
    if (bad) { atomicExch(overflow, 1u); }
  }
}

// qq[q] = |q|^2 in the order of the exact scores (coordinate 0 to d - 1, every operation rounded on its own): a chain of d
// dependent additions per query. Made by one thread of the verification it kept a whole block waiting; here 32 queries share
// a warp, their coordinates come through shared memory in pieces of 32, and the chains run side by side.
template <typename T>
__global__ void __launch_bounds__(32) query_sqnorm_kernel(const uint8_t* queries, size_t qpitch, int d, int64_t nq, double* qq)
{
  __shared__ float tile[32][33];
  const int lane   = threadIdx.x;
  const int64_t q0 = static_cast<int64_t>(blockIdx.x) * 32;
  const int n      = static_cast<int>(min(static_cast<int64_t>(32), nq - q0));
  double a         = 0;
  float next[32];  // the piece after this one, on its way while this one is summed
  auto fetch = [&](int t) {
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      const T* row = reinterpret_cast<const T*>(queries + static_cast<size_t>(q0 + i) * qpitch);
      next[i]      = i < n && t + lane < d ? static_cast<float>(row[t + lane]) : 0.f;
    }
  };
  fetch(0);
  for (int t0 = 0; t0 < d; t0 += 32) {
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 32; ++i) { tile[i][lane] = next[i]; }
    __syncwarp();
    if (t0 + 32 < d) { fetch(t0 + 32); }
#pragma unroll
    for (int i = 0; i < 32; ++i) {  // beyond the last coordinate zeros are added, which leave the sum as it is
      const double v = static_cast<double>(tile[lane][i]);
      a              = __dadd_rn(a, __dmul_rn(v, v));
    }
  }
  if (lane < n) { qq[q0 + lane] = a; }
}

/// The float of a key of the screen kernel's float_key, and a value less half a query's allowance, rounded down.
__device__ __forceinline__ float float_of_key(int32_t key) { return __int_as_float(key ^ ((key >> 31) & 0x7fffffff)); }
__device__ __forceinline__ float lowered(float v, float shift) { return __fadd_rd(v, -__fmul_ru(0.5f, shift)); }
__device__ __forceinline__ int32_t lowered_bits(float v, float shift) { return __float_as_int(lowered(v, shift)); }

// fp16 codes, in two steps around the optional exchange of thresholds between shards. Step 0: thr[q] = the key of the
// k-th largest group maximum (see float_key in the screen kernel) -> the key of value - shift[q] / 2, a score that k
// rows of this index certainly reach in exact arithmetic. Step 1: such a key -> float bits of the screen's
// threshold, bound - shift[q] / 2. Both subtractions round down. (Without an exchange kth_largest_kernel makes both.)
__global__ void finish_thr_f16_kernel(int32_t* thr, const float* shift, int nq, int step, int per)
{
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= nq) { return; }
  const int32_t b = lowered_bits(float_of_key(thr[q]), shift[q / per]);
  thr[q]          = step == 0 ? (b ^ ((b >> 31) & 0x7fffffff)) : b;
}

__global__ void chain_max_f32_kernel(const float* init, int64_t c0, int64_t n, float* cmax)
{
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) { return; }
  float m = -CUDART_INF_F;
  for (int k = 0; k < 16; ++k) { m = fmaxf(m, init[(c0 + i) * 16 + k]); }
  cmax[c0 + i] = m;
}

// The rows of candidate lists, one thread per chain.
__global__ void candidate_rows_kernel(const Candidate* cand, const uint32_t* cnt, uint32_t cap, int64_t n_rows,
                                      uint32_t* row_cnt, int32_t* rows, uint32_t row_cap)
{
  const uint32_t n = min(cnt[blockIdx.x], cap);
  for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
    const Candidate c = cand[static_cast<size_t>(blockIdx.x) * cap + i];
    for (uint32_t mask = c.mask; mask; mask &= mask - 1) {
      const int64_t r = static_cast<int64_t>(c.chain) * kChainRows + __ffs(mask) - 1;
      if (r < n_rows) {
        const uint32_t at = atomicAdd(row_cnt + blockIdx.x, 1u);
        if (at < row_cap) { rows[static_cast<size_t>(blockIdx.x) * row_cap + at] = static_cast<int32_t>(r); }
      }
    }
  }
}

// A warp per row of the tail. Its code stays in the lanes' registers as far as it fits (16 bytes a lane: 512 bytes) while the
// queries of its label pass by; their codes come from L2. The sum of a float pair is made of 32 partial sums and a tree, far
// inside the bound of the tensor cores' sums that the thresholds allow for.
template <int KIND>
__global__ void tail_kernel(TailRows t, const uint8_t* q_codes, const int32_t* thr, const int32_t* label, const int32_t* slot0,
                            const int32_t* n_slots, int n_runs, Candidate* cand, uint32_t* cnt, uint32_t cap, int ld)
{
  const int lane = threadIdx.x & 31;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < t.n_tail; i += warps) {
    const int32_t id = t.tail_id0 + i;
    if (t.removed[id]) { continue; }
    const int32_t l = t.row_labels[id];
    int lo = 0, hi = n_runs - 1;  // first run whose label is not below l
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (label[mid] < l) {
        lo = mid + 1;
      } else {
        hi = mid;
      }
    }
    if (l < 0 || label[lo] != l) { continue; }
    const int32_t row  = t.inv[id];
    const int32_t e    = t.init[row];
    const uint4* x     = reinterpret_cast<const uint4*>(t.codes + static_cast<size_t>(row) * t.code_pitch);
    const int n_vec    = static_cast<int>(t.code_pitch / 16);
    const uint4 zero   = make_uint4(0, 0, 0, 0);
    const uint4 x0     = lane < n_vec ? __ldg(x + lane) : zero;
    auto add = [](const uint4& a, const uint4& b, int& isum, float& fsum) {
      const uint32_t u[4] = {a.x, a.y, a.z, a.w}, v[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if constexpr (KIND == 2) {
          const float2 p = __half22float2(*reinterpret_cast<const __half2*>(&u[j]));
          const float2 q = __half22float2(*reinterpret_cast<const __half2*>(&v[j]));
          fsum           = fmaf(p.x, q.x, fsum);
          fsum           = fmaf(p.y, q.y, fsum);
        } else if constexpr (KIND == 1) {
          isum = __dp4a(static_cast<int>(u[j]), static_cast<int>(v[j]), isum);
        } else {
          isum = static_cast<int>(__dp4a(u[j], v[j], static_cast<unsigned>(isum)));
        }
      }
    };
    const int s1 = slot0[lo] + n_slots[lo];
    for (int s = slot0[lo]; s < s1; ++s) {
      const uint4* q = reinterpret_cast<const uint4*>(q_codes + static_cast<size_t>(s) * t.code_pitch);
      int isum       = 0;
      float fsum     = 0;
      if (lane < n_vec) { add(x0, __ldg(q + lane), isum, fsum); }
      for (int c = lane + 32; c < n_vec; c += 32) { add(__ldg(x + c), __ldg(q + c), isum, fsum); }
      int32_t value;
      bool hit;
      if constexpr (KIND == 2) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) { fsum += __shfl_xor_sync(0xffffffffu, fsum, o); }
        const float v = fsum + __int_as_float(e);
        value         = __float_as_int(v);
        hit           = v >= __int_as_float(thr[s]);
      } else {
        value = __reduce_add_sync(0xffffffffu, isum) + e;
        hit   = value >= thr[s];
      }
      if (lane == 0 && hit) {
        const uint32_t at = atomicAdd(cnt + s, 1u);
        if (at < cap) {
          const int64_t r = t.n_rows + i;  // n_rows is a multiple of the chain length
          reinterpret_cast<uint4*>(cand)[static_cast<size_t>(s) * ld + at] =
            make_uint4(static_cast<uint32_t>(r / kChainRows), 1u << (r % kChainRows), static_cast<uint32_t>(value), 0u);
        }
      }
    }
  }
}

// rows [q, 0 : n_parts * k] = the lists parts[p, q, 0:k] of every part side by side.
__global__ void union_rows_kernel(const int32_t* parts, int n_parts, int nq, int k, int32_t* rows, int64_t ld)
{
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int m     = n_parts * k;
  if (i >= static_cast<int64_t>(nq) * m) { return; }
  const int64_t q = i / m;
  const int c     = static_cast<int>(i % m), part = c / k, j = c % k;
  rows[q * ld + c] = parts[(static_cast<int64_t>(part) * nq + q) * k + j];
}

// Block per query: the k-th largest of ng int32 values by a most-significant-digit radix walk. The row is copied to
// shared memory first when it fits (vals != global row).
// With ng_rows the rows have their own lengths; a negative length marks a row without a query: thr = never.
// Every thread of the block: out [k] = the k largest of row[0:ng] (any order) given their k-th, t: the values above it,
// then copies of it. (Which k of several equal values are meant does not matter to a threshold.) *counter is shared.
__device__ void emit_topk(const int32_t* row, int ng, int32_t t, int k, int32_t* out, uint32_t* counter)
{
  __syncthreads();
  if (threadIdx.x == 0) { *counter = 0; }
  __syncthreads();
  for (int i = threadIdx.x; i < ng; i += blockDim.x) {
    const int32_t v = row[i];
    if (v > t) {
      const uint32_t pos = atomicAdd(counter, 1u);
      if (pos < static_cast<uint32_t>(k)) { out[pos] = v; }  // fewer than k values lie above the k-th largest
    }
  }
  __syncthreads();
  for (int i = static_cast<int>(min(*counter, static_cast<uint32_t>(k))) + threadIdx.x; i < k; i += blockDim.x) { out[i] = t; }
}

// With topk [nq, k] the k largest values of every row are written there as well (emit_topk). With shift [nq] (fp16 codes) the
// threshold is lowered by it and leaves as float bits (both steps of finish_thr_f16_kernel); zero [nq] is set to 0: what follows
// counts in it.
__global__ void __launch_bounds__(512, 4) kth_largest_kernel(const int32_t* gmax, int64_t ld, int ng, int k, int32_t* thr,
                                                              int in_smem, const int32_t* ng_rows, int32_t never, int32_t* topk,
                                                              const float* shift, uint32_t* zero)
{
  extern __shared__ int32_t row_smem[];
  __shared__ uint32_t hist[256];
  __shared__ uint32_t s_prefix, s_remaining;
  // the k-th largest value of the row -> its threshold
  auto answer = [&](int32_t t) {
    if (threadIdx.x != 0) { return; }
    if (shift) { t = lowered_bits(lowered(float_of_key(t), shift[blockIdx.x]), shift[blockIdx.x]); }
    thr[blockIdx.x] = t;
    if (zero) { zero[blockIdx.x] = 0; }
  };
  const int32_t* row = gmax + static_cast<int64_t>(blockIdx.x) * ld;
  int32_t* topk_row  = topk ? topk + static_cast<int64_t>(blockIdx.x) * k : nullptr;
  if (ng_rows) {
    ng = ng_rows[blockIdx.x];
    if (ng < 0) {
      answer(never);
      if (topk_row) {
        for (int i = threadIdx.x; i < k; i += blockDim.x) { topk_row[i] = never; }
      }
      return;
    }
  }
  if (ng < k) {
    answer(static_cast<int32_t>(0x80000000u));
    if (topk_row) {
      for (int i = threadIdx.x; i < k; i += blockDim.x) { topk_row[i] = static_cast<int32_t>(0x80000000u); }
    }
    return;
  }
  // The row goes to shared memory (when it fits) and its smallest and largest key are found on the way: the radix walk
  // then runs on key - smallest and starts at the highest byte in which the keys differ. Group maxima of one query lie
  // close together; walking all 32 bits would put nearly every value into one bin of the first passes, and the
  // shared-memory atomics on that bin would serialise.
  __shared__ uint32_t s_lo, s_hi;
  if (threadIdx.x == 0) {
    s_lo = 0xffffffffu;
    s_hi = 0u;
  }
  __syncthreads();
  uint32_t lo = 0xffffffffu, hi = 0u;
  auto see = [&](int32_t v) {
    const uint32_t key = static_cast<uint32_t>(v) ^ 0x80000000u;
    lo                 = min(lo, key);
    hi                 = max(hi, key);
  };
  if (in_smem) {
    const int n4 = ng >> 2;  // rows start 16-byte aligned (ld is a multiple of 8)
    for (int i = threadIdx.x; i < n4; i += blockDim.x) {
      const int4 v                         = __ldg(reinterpret_cast<const int4*>(row) + i);
      reinterpret_cast<int4*>(row_smem)[i] = v;
      see(v.x), see(v.y), see(v.z), see(v.w);
    }
    for (int i = (n4 << 2) + threadIdx.x; i < ng; i += blockDim.x) {
      row_smem[i] = row[i];
      see(row_smem[i]);
    }
    row = row_smem;
  } else {
    for (int i = threadIdx.x; i < ng; i += blockDim.x) { see(row[i]); }
  }
  const uint32_t my_hi = hi;  // the largest key this thread saw (0: none)
  // Small k: the k-th largest of the maxima of G groups of threads is a value that k elements reach (the k groups at
  // or above it hold one each), so only the few elements at or above it can be the k-th largest of the row: they are
  // collected in one more pass over the row and ranked by counting. No histogram, no contended atomics. When the list
  // does not hold them (many equal values), the radix walk below takes over.
  constexpr int kCollect = 1024;
  __shared__ uint32_t s_group[512], s_list[kCollect];
  __shared__ uint32_t s_bound, s_count, s_answer;
  const int n_threads = blockDim.x;
  if (in_smem && (n_threads == 512 || n_threads == 256 || n_threads == 128) && 2 * k <= n_threads) {
    int groups = 16;
    while (groups < 2 * k) { groups <<= 1; }
    const int per_group = n_threads / groups;  // 32, 16, ..., 1 threads
    uint32_t g_hi       = my_hi;
    for (int o = 1; o < per_group; o <<= 1) { g_hi = max(g_hi, __shfl_xor_sync(0xffffffffu, g_hi, o)); }
    if ((threadIdx.x & (per_group - 1)) == 0) { s_group[threadIdx.x / per_group] = g_hi; }
    if (threadIdx.x == 0) { s_count = 0; }
    __syncthreads();
    if (threadIdx.x < groups) {
      const uint32_t u = s_group[threadIdx.x];
      int rank         = 0;
      for (int j = 0; j < groups; ++j) {
        const uint32_t v = s_group[j];
        rank += (v > u || (v == u && j < static_cast<int>(threadIdx.x))) ? 1 : 0;
      }
      if (rank == k - 1) { s_bound = u; }
    }
    __syncthreads();
    const uint32_t bound = s_bound;
    for (int i = threadIdx.x; i < ng; i += n_threads) {
      const uint32_t key = static_cast<uint32_t>(row[i]) ^ 0x80000000u;
      if (key >= bound) {
        const uint32_t pos = atomicAdd(&s_count, 1u);
        if (pos < kCollect) { s_list[pos] = key; }
      }
    }
    __syncthreads();
    const int n_list = static_cast<int>(s_count);
    if (n_list <= kCollect) {  // n_list >= k: the k group maxima at or above the bound are k elements of the row
      for (int i = threadIdx.x; i < n_list; i += n_threads) {
        const uint32_t u = s_list[i];
        int greater = 0, at_least = 0;
        for (int j = 0; j < n_list; ++j) {
          const uint32_t v = s_list[j];
          greater += v > u ? 1 : 0;
          at_least += v >= u ? 1 : 0;
        }
        if (greater < k && k <= at_least) { s_answer = u; }  // every thread that gets here holds the same value
      }
      __syncthreads();
      const int32_t t = static_cast<int32_t>(s_answer ^ 0x80000000u);
      answer(t);
      if (topk_row) { emit_topk(row, ng, t, k, topk_row, &s_count); }
      return;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMin(&s_lo, lo);
    atomicMax(&s_hi, hi);
  }
  __syncthreads();
  const uint32_t base  = s_lo;
  const uint32_t range = s_hi - base;
  const int top        = range == 0u ? 0 : 32 - __clz(range);  // bits in which key - base can be set
  uint32_t prefix = 0, mask = 0, remaining = static_cast<uint32_t>(k);
  for (int shift = ((top + 7) / 8 - 1) * 8; shift >= 0; shift -= 8) {
    for (int i = threadIdx.x; i < 256; i += blockDim.x) { hist[i] = 0; }
    __syncthreads();
    for (int i = threadIdx.x; i < ng; i += blockDim.x) {
      const uint32_t key = (static_cast<uint32_t>(row[i]) ^ 0x80000000u) - base;
      if ((key & mask) == prefix) { atomicAdd(&hist[(key >> shift) & 255u], 1u); }
    }
    __syncthreads();
    if (threadIdx.x < 32) {
      // bucket b (from the top) where the running count reaches `remaining`: warp scan over 8 buckets per lane
      const int lane = threadIdx.x;
      uint32_t c[8], sum = 0;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        c[i] = hist[255 - (lane * 8 + i)];
        sum += c[i];
      }
      uint32_t incl = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) { incl += v; }
      }
      const uint32_t before = incl - sum;
      const bool mine       = before < remaining && incl >= remaining;
      if (mine) {
        uint32_t cum = before;
        int i        = 0;
        for (; i < 7; ++i) {
          if (cum + c[i] >= remaining) { break; }
          cum += c[i];
        }
        s_prefix    = prefix | (static_cast<uint32_t>(255 - (lane * 8 + i)) << shift);
        s_remaining = remaining - cum;
      }
    }
    __syncthreads();
    prefix    = s_prefix;
    remaining = s_remaining;
    mask |= 0xffu << shift;
  }
  const int32_t t = static_cast<int32_t>((prefix + base) ^ 0x80000000u);
  answer(t);
  if (topk_row) { emit_topk(row, ng, t, k, topk_row, &s_count); }
}

// The same thresholds for short rows and k > 32, a warp to a row of up to 32 kBitsHeld values: they stay in registers, and the
// largest bound that k of them reach is found bit by bit from the highest bit in which they differ. kth_largest_kernel compares
// the maxima of 2k groups of threads with one another, for such a row every value with every other, and is bound by those
// instructions (16 384 rows of 244 values, k = 100: 315 us; this one 31 us). Small k is cheap there (1000 rows of 520 values,
// k = 10: a call 171 us, with this kernel and 32 values a lane 180 us), and with several warps to a row every bit costs a step of
// the whole block (8192 values: 21 us there, 31 us). Lists of the k largest, for an exchange between shards, are made there too.
constexpr int kBitsHeld = 16;
__global__ void __launch_bounds__(128) kth_bits_kernel(const int32_t* gmax, int64_t ld, int n_rows, int ng, int k, int32_t* thr,
                                                       const int32_t* ng_rows, int32_t never, const float* shift, uint32_t* zero)
{
  const int lane = threadIdx.x & 31;
  const int q    = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (q >= n_rows) { return; }  // warps are independent
  auto answer = [&](int32_t t) {
    if (lane != 0) { return; }
    if (shift) { t = lowered_bits(lowered(float_of_key(t), shift[q]), shift[q]); }
    thr[q] = t;
    if (zero) { zero[q] = 0; }
  };
  if (ng_rows) {
    ng = ng_rows[q];
    if (ng < 0) {
      answer(never);
      return;
    }
  }
  if (ng < k) {
    answer(static_cast<int32_t>(0x80000000u));
    return;
  }
  // the values as unsigned keys; 0 beyond the row's end, which no bound tried below lets through
  const int32_t* row = gmax + static_cast<int64_t>(q) * ld;
  uint32_t u[kBitsHeld], lo = 0xffffffffu, hi = 0;
#pragma unroll
  for (int i = 0; i < kBitsHeld; ++i) {
    const int at = lane + i * 32;
    u[i]         = 0;
    if (at < ng) {
      u[i] = static_cast<uint32_t>(__ldg(row + at)) ^ 0x80000000u;
      lo   = min(lo, u[i]);
      hi   = max(hi, u[i]);
    }
  }
  lo = __reduce_min_sync(0xffffffffu, lo);
  hi = __reduce_max_sync(0xffffffffu, hi);
  const int top = lo == hi ? 0 : 32 - __clz(lo ^ hi);  // bits from here up are those of all values
  uint32_t t    = top == 32 ? 0u : hi >> top << top;
  for (int bit = top - 1; bit >= 0; --bit) {
    const uint32_t next = t | (1u << bit);
    int reach           = 0;
#pragma unroll
    for (int i = 0; i < kBitsHeld; ++i) { reach += u[i] >= next ? 1 : 0; }
    if (__reduce_add_sync(0xffffffffu, reach) >= k) { t = next; }
  }
  answer(static_cast<int32_t>(t ^ 0x80000000u));
}

// Warp per query: the k-th largest of the n_parts * k values parts[p, q, 0:k], p < n_parts, by counting ranks
// (m = n_parts * k <= kUnionMax). Shared memory: m ints per warp.
constexpr int kUnionMax = 512;
__global__ void union_kth_kernel(const int32_t* parts, int n_parts, int nq, int k, int32_t* thr)
{
  extern __shared__ int32_t union_smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int q    = blockIdx.x * (blockDim.x >> 5) + warp;
  if (q >= nq) { return; }  // warps are independent: no block-wide barrier below
  const int m = n_parts * k;
  int32_t* v  = union_smem + warp * m;
  for (int i = lane; i < m; i += 32) { v[i] = parts[(static_cast<int64_t>(i / k) * nq + q) * k + (i % k)]; }
  __syncwarp();
  for (int i = lane; i < m; i += 32) {
    const int32_t x = v[i];
    int rank        = 0;
    for (int j = 0; j < m; ++j) {
      const int32_t y = v[j];
      rank += (y > x || (y == x && j < i)) ? 1 : 0;
    }
    if (rank == k - 1) { thr[q] = x; }  // ranks are a permutation of 0 .. m - 1: exactly one element
  }
}

// Exact scores of 8-bit rows against an 8-bit query in integer arithmetic: <q, x> and |x|^2 by 4-way byte dot products
// (int32 is enough: 255^2 * 4096 < 2^31), the score |q|^2 + |x|^2 - 2 <q, x> (L2) or |q|^2 - 2 <q, x> in int64. Every
// partial sum of the fp64 loop over the coordinates is an integer below 2^53, so that loop returns this very integer:
// the results are bit-identical, without one conversion to double per coordinate. |score| < 2^31.
// A row is spread over kRowLanes adjacent lanes of a warp: lane `sub` takes the 16-byte pieces sub, sub + 8, ..., so
// that the lanes of a row read one 128-byte line together and a warp's load covers four whole lines; the partial sums
// are added across the lanes by shuffles (integers: exact in any order). kRowUnroll rows per lane group are in flight
// at once. Every lane of the warp must call it; row < 0 = no row. The results are valid in all lanes of a row.
// qb: the query's bytes in shared memory, zero padded to whole 16-byte vectors like the stored rows.
constexpr int kRowLanes  = 8;
constexpr int kRowUnroll = 4;
template <typename T, int METRIC>
__device__ __forceinline__ void int_row_scores(const uint8_t* vectors, size_t pitch, const int32_t (&row)[kRowUnroll], int d,
                                               const uint4* qb, long long qq, int sub, long long (&score)[kRowUnroll])
{
  const int n_vec = (d + 15) / 16;
  int ip[kRowUnroll], xx[kRowUnroll];
  const uint4* p[kRowUnroll];
#pragma unroll
  for (int u = 0; u < kRowUnroll; ++u) {
    ip[u] = 0, xx[u] = 0;
    p[u] = reinterpret_cast<const uint4*>(vectors + static_cast<size_t>(max(row[u], 0)) * pitch);
  }
  for (int c = sub; c < n_vec; c += kRowLanes) {
    const uint4 a = qb[c];
    uint4 w[kRowUnroll];
#pragma unroll
    for (int u = 0; u < kRowUnroll; ++u) { w[u] = row[u] >= 0 ? __ldg(p[u] + c) : make_uint4(0, 0, 0, 0); }
#pragma unroll
    for (int u = 0; u < kRowUnroll; ++u) {
      if constexpr (std::is_same<T, int8_t>::value) {
        ip[u] = __dp4a(static_cast<int>(w[u].x), static_cast<int>(a.x), ip[u]);
        ip[u] = __dp4a(static_cast<int>(w[u].y), static_cast<int>(a.y), ip[u]);
        ip[u] = __dp4a(static_cast<int>(w[u].z), static_cast<int>(a.z), ip[u]);
        ip[u] = __dp4a(static_cast<int>(w[u].w), static_cast<int>(a.w), ip[u]);
        if constexpr (METRIC == kL2) {
          xx[u] = __dp4a(static_cast<int>(w[u].x), static_cast<int>(w[u].x), xx[u]);
          xx[u] = __dp4a(static_cast<int>(w[u].y), static_cast<int>(w[u].y), xx[u]);
          xx[u] = __dp4a(static_cast<int>(w[u].z), static_cast<int>(w[u].z), xx[u]);
          xx[u] = __dp4a(static_cast<int>(w[u].w), static_cast<int>(w[u].w), xx[u]);
        }
      } else {
        ip[u] = static_cast<int>(__dp4a(w[u].x, a.x, static_cast<unsigned>(ip[u])));
        ip[u] = static_cast<int>(__dp4a(w[u].y, a.y, static_cast<unsigned>(ip[u])));
        ip[u] = static_cast<int>(__dp4a(w[u].z, a.z, static_cast<unsigned>(ip[u])));
        ip[u] = static_cast<int>(__dp4a(w[u].w, a.w, static_cast<unsigned>(ip[u])));
        if constexpr (METRIC == kL2) {
          xx[u] = static_cast<int>(__dp4a(w[u].x, w[u].x, static_cast<unsigned>(xx[u])));
          xx[u] = static_cast<int>(__dp4a(w[u].y, w[u].y, static_cast<unsigned>(xx[u])));
          xx[u] = static_cast<int>(__dp4a(w[u].z, w[u].z, static_cast<unsigned>(xx[u])));
          xx[u] = static_cast<int>(__dp4a(w[u].w, w[u].w, static_cast<unsigned>(xx[u])));
        }
      }
    }
  }
#pragma unroll
  for (int u = 0; u < kRowUnroll; ++u) {
#pragma unroll
    for (int o = 1; o < kRowLanes; o <<= 1) {
      ip[u] += __shfl_xor_sync(0xffffffffu, ip[u], o);
      if constexpr (METRIC == kL2) { xx[u] += __shfl_xor_sync(0xffffffffu, xx[u], o); }
    }
    score[u] = qq + static_cast<long long>(xx[u]) - 2ll * static_cast<long long>(ip[u]);
  }
}

// Every thread of the block: the k-th largest of n keys in shared memory, 1 <= k <= number of keys that are not 0 (0: no
// key). Up to 512 keys: one warp holds them in registers and finds the largest threshold that k of them reach bit by bit,
// without a step of the whole block in between. More: a most-significant-digit radix walk that starts at the highest byte in
// which the keys differ. `scratch`: 260 words.
__device__ uint32_t block_kth_largest(const uint32_t* key, int n, int k, uint32_t* scratch)
{
  const int n_threads = blockDim.x;
  constexpr int kHeld = 16;
  if (n <= 32 * kHeld) {
    if (threadIdx.x < 32) {
      uint32_t u[kHeld];
      uint32_t hi = 0;
#pragma unroll
      for (int i = 0; i < kHeld; ++i) {
        const int at = threadIdx.x + i * 32;
        u[i]         = at < n ? key[at] : 0u;
        hi           = max(hi, u[i]);
      }
      hi         = __reduce_max_sync(0xffffffffu, hi);
      uint32_t t = 0;
      bool exact = false;
      for (int bit = 31 - __clz(hi); bit >= 0 && !exact; --bit) {
        const uint32_t next = t | (1u << bit);
        int reach           = 0;
#pragma unroll
        for (int i = 0; i < kHeld; ++i) { reach += u[i] >= next ? 1 : 0; }
        reach = __reduce_add_sync(0xffffffffu, reach);
        if (reach >= k) { t = next; }
        exact = reach == k;
      }
      uint32_t least = 0xffffffffu;  // the smallest key that reaches t
#pragma unroll
      for (int i = 0; i < kHeld; ++i) { least = u[i] >= t && u[i] != 0u ? min(least, u[i]) : least; }
      least = __reduce_min_sync(0xffffffffu, least);
      if (threadIdx.x == 0) { scratch[256] = least; }
    }
    __syncthreads();
    return scratch[256];
  }
  uint32_t lo = 0xffffffffu, hi = 0u;
  for (int i = threadIdx.x; i < n; i += n_threads) {
    const uint32_t v = key[i];
    if (v != 0u) { lo = min(lo, v), hi = max(hi, v); }
  }
  lo = __reduce_min_sync(0xffffffffu, lo);
  hi = __reduce_max_sync(0xffffffffu, hi);
  if (threadIdx.x == 0) { scratch[257] = 0xffffffffu, scratch[258] = 0u; }
  __syncthreads();
  if ((threadIdx.x & 31) == 0) {
    atomicMin(scratch + 257, lo);
    atomicMax(scratch + 258, hi);
  }
  __syncthreads();
  const uint32_t base  = scratch[257];
  const uint32_t range = scratch[258] - base;
  const int top        = range == 0u ? 0 : 32 - __clz(range);
  uint32_t prefix = 0, mask = 0, remaining = static_cast<uint32_t>(k);
  for (int shift = ((top + 7) / 8 - 1) * 8; shift >= 0; shift -= 8) {
    for (int i = threadIdx.x; i < 256; i += n_threads) { scratch[i] = 0; }
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += n_threads) {
      const uint32_t v = key[i];
      if (v != 0u && ((v - base) & mask) == prefix) { atomicAdd(&scratch[((v - base) >> shift) & 255u], 1u); }
    }
    __syncthreads();
    if (threadIdx.x < 32) {
      const int lane = threadIdx.x;
      uint32_t c[8], sum = 0;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        c[i] = scratch[255 - (lane * 8 + i)];
        sum += c[i];
      }
      uint32_t incl = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) { incl += v; }
      }
      const uint32_t before = incl - sum;
      if (before < remaining && incl >= remaining) {
        uint32_t cum = before;
        int i        = 0;
        for (; i < 7; ++i) {
          if (cum + c[i] >= remaining) { break; }
          cum += c[i];
        }
        scratch[257] = prefix | (static_cast<uint32_t>(255 - (lane * 8 + i)) << shift);
        scratch[258] = remaining - cum;
      }
    }
    __syncthreads();
    prefix    = scratch[257];
    remaining = scratch[258];
    mask |= 0xffu << shift;
  }
  __syncthreads();
  return prefix + base;
}

// Sorts m entries in shared memory by (score, id), ascending, in place. Up to one entry per thread: every entry's place
// is the number of entries before it (the ids are distinct); more: bitonic, the tail up to next_pow2(m) filled up.
template <typename IdT>
__device__ void sort_pairs(double* s, IdT* id, int m)
{
  __syncthreads();
  if (m <= static_cast<int>(blockDim.x)) {
    double x = 0;
    IdT xi   = 0;
    int place = 0;
    const bool mine = static_cast<int>(threadIdx.x) < m;
    if (mine) {
      x  = s[threadIdx.x];
      xi = id[threadIdx.x];
      for (int j = 0; j < m; ++j) { place += pair_less(s[j], id[j], x, xi) ? 1 : 0; }
    }
    __syncthreads();
    if (mine) {
      s[place]  = x;
      id[place] = xi;
    }
    __syncthreads();
    return;
  }
  const int n2 = next_pow2(m);
  for (int i = m + threadIdx.x; i < n2; i += blockDim.x) {
    s[i]  = CUDART_INF;
    id[i] = static_cast<IdT>(0x7fffffff);
  }
  bitonic_sort(s, id, n2);
}

// The same for distinct 64-bit keys.
__device__ void sort_keys(unsigned long long* key, int m)
{
  __syncthreads();
  if (m <= static_cast<int>(blockDim.x)) {
    unsigned long long x = 0;
    int place            = 0;
    const bool mine      = static_cast<int>(threadIdx.x) < m;
    if (mine) {
      x = key[threadIdx.x];
      for (int j = 0; j < m; ++j) { place += key[j] < x ? 1 : 0; }
    }
    __syncthreads();
    if (mine) { key[place] = x; }
    __syncthreads();
    return;
  }
  const int n2 = next_pow2(m);
  for (int i = m + threadIdx.x; i < n2; i += blockDim.x) { key[i] = ~0ull; }
  bitonic_sort_keys(key, n2);
}

// ------------------------------------------------------------------------------------------- stored |x|^2 (cosine)
// Warp per 32 consecutive rows: out[r] = the sum over the coordinates, in order, of x_t^2 in fp64 with every product and
// every sum rounded on its own: bit for bit the sum the cosine verification makes for a candidate row (Acc). The rows
// come through a shared-memory tile as in verify_select_kernel, so that the loads cover whole lines.
constexpr int kSqnormStride = 144;
template <typename T>
__global__ void __launch_bounds__(128) row_sqnorm_kernel(const uint8_t* vectors, size_t pitch, int d, int64_t n, double* out)
{
  __shared__ __align__(16) uint8_t tiles[4 * 32 * kSqnormStride];
  constexpr int V    = Elems<T>::kPerVec;
  const int lane     = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t row0 = (static_cast<int64_t>(blockIdx.x) * 4 + warp) * 32;
  if (row0 >= n) { return; }  // warps are independent: no block-wide barrier below
  uint8_t* tile      = tiles + warp * 32 * kSqnormStride;
  const int piece = lane & 7, row_in_load = lane >> 3;
  const int n_pieces = static_cast<int>((static_cast<size_t>(d) * sizeof(T) + 15) / 16);  // rows are zero padded to the pitch
  const int64_t mine = row0 + lane;
  double xx          = 0;
  for (int p0 = 0; p0 < n_pieces; p0 += 8) {
    uint4 w[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int64_t r = row0 + 4 * j + row_in_load;
      w[j] = (r < n && p0 + piece < n_pieces) ? __ldg(reinterpret_cast<const uint4*>(vectors + static_cast<size_t>(r) * pitch) + p0 + piece)
                                              : make_uint4(0, 0, 0, 0);
    }
    __syncwarp();  // every lane is done with the slab before
#pragma unroll
    for (int j = 0; j < 8; ++j) { *reinterpret_cast<uint4*>(tile + (4 * j + row_in_load) * kSqnormStride + piece * 16) = w[j]; }
    __syncwarp();
    if (mine < n) {
      const int np = min(8, n_pieces - p0);
      for (int p = 0; p < np; ++p) {
        const uint4 x4 = *reinterpret_cast<const uint4*>(tile + lane * kSqnormStride + p * 16);
        double x[V];
        Elems<T>::unpack(x4, x);
        const int t0 = (p0 + p) * V;
        for (int e = 0; e < V && t0 + e < d; ++e) { xx = __dadd_rn(xx, __dmul_rn(x[e], x[e])); }
      }
    }
  }
  if (mine < n) { out[mine] = xx; }
}

// ------------------------------------------------------------------------------------------- verify + select
// Staging tiles of the float rows: per warp 32 rows of a 128-byte slab, 144 bytes apart (a lane's 16-byte reads of its
// own row then fall on distinct banks within every quarter warp).
constexpr int kStageStride = 144;
__device__ __forceinline__ uint8_t* stage_of(void* after_the_arrays)
{
  return reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(after_the_arrays) + 15) & ~static_cast<uintptr_t>(15));
}
// Block per query. A candidate chain comes with its largest product, so the candidates are ranked before a vector is read.
// With value = product + e of the row (what the thresholds are made of), a chain whose kept rows may all be returned has a
// row of value >= product + the smallest e of them; a row of it has a value <= product + its own e (the same number when
// the chain kept one row, as nearly all do). Let v_k be the k-th largest of the former over the chains (rows of k
// different chains reach it). Only rows whose latter can still belong to the k nearest are scored in fp64:
//   8-bit vectors  those >= v_k. Values are exact but for the bit that e = -floor(|x|^2 / 2) drops: 2 value - 1 or 2 value
//                  is the exact term, and twice a value below v_k lies below 2 v_k - 1, which k rows reach.
//   fp16 codes     those >= v_k - shift, shift = twice the most a value may be off (see encode_f16_queries_kernel): k rows
//                  certainly reach v_k - shift / 2, and a row that does has a value of at least v_k - shift.
// Reading and scoring rows is what bounds the kernel (d coordinates of a gathered row per candidate, each with two or
// three fp64 operations), and the screen keeps several times k candidates; after the ranking about k are left:
// 10 000 queries, k = 100, 1 M x 768 float coordinates: 220 of 619 rows, 5.96 -> 2.27 ms; 777 queries, k = 33, 1.2 M x 100
// bytes with a bitset: 34 of 1017 rows, 138 + 67 us (the launch that made lists of rows) -> 64 us; 1000 queries, k = 10,
// 100 000 x 128 floats: 14 of 209 rows, 69 + 12 -> 25 us.
// Dynamic shared memory: the query (doubles, or bytes) | sc [n2] doubles | id [n2] int32, n2 = next_pow2(cap); for 8-bit
// rows n2 64-bit keys in place of sc. Before the scores are made the space of sc holds the rows' values and ids, and the
// space of id what the chains reach.
template <typename T>
constexpr bool kByteRows = std::is_same<T, int8_t>::value || std::is_same<T, uint8_t>::value;
// |q|^2 as the scores have it, by one thread.
template <typename T>
__device__ double query_sqnorm(const Candidates& cd, const void* queries, size_t qpitch, int d, int q)
{
  if constexpr (kByteRows<T>) {
    const T* src = reinterpret_cast<const T*>(static_cast<const uint8_t*>(queries) + static_cast<size_t>(q) * qpitch);
    int a        = 0;
    for (int t = 0; t < d; ++t) { a += static_cast<int>(src[t]) * static_cast<int>(src[t]); }
    return a;
  } else {
    return cd.qq[q];
  }
}

// One thread reports an overflowed query with the tighter threshold that the k-th best exact score `kth` among the listed
// candidates gives (+inf: fewer than k). qq: |q|^2, where the metric's scores have a use for it.
template <typename T, int METRIC>
__device__ void report_overflow(const Refine& rf, int q, int qb, const void* queries, size_t qpitch, int d, double qq, double kth,
                                int32_t* ovf_list, unsigned int* ovf_count)
{
  const unsigned int pos = atomicAdd(ovf_count, 1u);
  ovf_list[pos]          = q;
  int32_t t              = rf.thr[qb];
  if (kth < CUDART_INF) {
    // the screen's value of a row as good as the k-th: <q, x> - |x|^2 / 2 (L2), <q, x> (inner product),
    // <q, x / |x|> (cosine)
    if (!kByteRows<T> && METRIC == kL2) {  // the scores had no use for it
      const uint8_t* src = static_cast<const uint8_t*>(queries) + static_cast<size_t>(q) * qpitch;
      for (int i = 0; i < d; ++i) {
        const double v = Elems<T>::one(src, i);
        qq             = __dadd_rn(qq, __dmul_rn(v, v));
      }
    }
    const double value = METRIC == kCos ? sqrt(qq) * (1.0 - 0.5 * kth) : 0.5 * (qq - kth);
    if (rf.kind == 1) {  // integer values: e = -floor(|x|^2 / 2) only raises a row's value
      const double cv  = ceil(value);
      const int32_t tv = cv >= 2147483647.0 ? 0x7fffffff : cv <= -2147483648.0 ? static_cast<int32_t>(0x80000000u)
                                                                                  : static_cast<int32_t>(cv);
      t = max(t, tv);
    } else {             // fp16 codes: the value the pass computes may be lower by half the query's allowance
      float f = __double2float_rd(value - 0.5 * static_cast<double>(rf.shift[q]));
      f       = nextafterf(f, -CUDART_INF_F);
      t       = __float_as_int(fmaxf(f, __int_as_float(t)));
    }
  }
  rf.thr2[pos] = t;
}

// The three steps (rank, score, sort) are one launch when the lists are short and the rows too. With longer lists (k > 256)
// scoring takes a block as many turns as lists are long, the blocks of a few hundred queries fill the GPU unevenly (1.15 waves
// of them for 512 queries) and those of a few queries leave it idle; with long rows (kLongRow bytes and more than 32 answers) a
// block holds the SM's shared memory through the steps in which it reads little, and the warps without 32 rows of their own
// wait for the others'. So there the steps are launches of their own: the rows to score are dealt out over the whole grid, and the
// lists are sorted by score intervals. The list of a query and its scores then lie in the memory of its candidates, which are
// no longer needed.
// 512 queries, k = 2048, 1 M x 128 halves (2402 rows a query): one launch 341 us; rank 38, score 97, sort 44 us.
// 10 000 queries, k = 100, 768 floats, 159 rows a query (labels): rank 108, score 945, sort 85 us, the call 2304 -> 2063 us;
// 220 rows a query: one launch 2316 us; rank 154, score 1516, sort 222 us.
enum : int { kFused = 0, kRank = 1, kScore = 2 };
constexpr int kSplitK  = 256;
constexpr int kLongRow = 1024;
template <typename T, int METRIC, bool STORED_XX, int PART>
__global__ void __launch_bounds__(PART == kRank || kByteRows<T> ? 1024 : 256, PART == kRank || kByteRows<T> ? 1 : 3)
verify_select_kernel(const uint8_t* vectors, size_t pitch, int d, const void* queries, size_t qpitch, int q0, Candidates cd,
                     int n2max, int k, Admit adm, double* best_s, int32_t* best_row, int32_t* ovf_list, unsigned int* ovf_count,
                     unsigned long long* stats, Refine rf, const int32_t* where, const double* sqnorm, int32_t* kept)
{
  extern __shared__ double sh[];
  __shared__ double s_qq;
  __shared__ uint32_t s_scratch[260];
  __shared__ int s_rows, s_sure, s_seen, s_kept;
  __shared__ long long s_qq_int;
  constexpr bool kBytes = kByteRows<T>;
  const int qb          = PART == kScore ? blockIdx.y : blockIdx.x;  // the query's number in its batch
  const int q           = q0 + qb;                                   // and in the call
  const int out         = cd.sel ? __ldg(cd.sel + q) : q;            // and its list of answers
  if (out < 0) {
    if (PART == kRank && threadIdx.x == 0) { kept[qb] = -1; }
    return;
  }
  const Candidate* mine = cd.cand + static_cast<size_t>(qb) * cd.ld;
  // split: the query's list and scores in the memory of its candidates (ld = n2max entries of 16 bytes)
  double* far_s    = reinterpret_cast<double*>(const_cast<Candidate*>(mine));
  int32_t* far_ids = reinterpret_cast<int32_t*>(far_s + n2max);
  double* qd   = sh;
  double* sc   = kBytes ? sh + (d + 15) / 16 * 2 : sh + d;  // fused: the scores and ids in shared memory
  int32_t* ids = reinterpret_cast<int32_t*>(sc + n2max);
  bool over    = false;
  int m        = 0;
  auto nothing = [&] {  // no candidate (a slot without a query, or nothing that the query may return)
    for (int t = threadIdx.x; t < k; t += blockDim.x) {
      best_s[static_cast<size_t>(out) * k + t]   = CUDART_INF;
      best_row[static_cast<size_t>(out) * k + t] = -1;
    }
  };
  auto give_up = [&] {
    if (threadIdx.x == 0) {
      ovf_list[atomicAdd(ovf_count, 1u)] = q;
      if (PART == kRank) { kept[qb] = -1; }
    }
  };
  if constexpr (PART == kScore) {
    const int32_t w = kept[qb];  // how many rows are scored; negative: the query was given up; bit 30: its list overflowed
    const int all   = w < 0 ? 0 : w & 0x3fffffff;
    // the rows in equal pieces of whole warps, but no fewer than the block's warps take at once
    const int each  = max(static_cast<int>(blockDim.x), ((all + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x) + 31) / 32 * 32);
    const int at    = static_cast<int>(blockIdx.x) * each;
    m               = min(each, all - at);
    if (m <= 0) { return; }
    sc  = far_s + at;
    ids = far_ids + at;
  }
  // A candidate list that overflowed (or more rows in it than the block holds): the query is reported in ovf_list. What the
  // block has are still rows at or above the query's threshold, and the k-th best exact score among them bounds the k-th
  // neighbour: a tighter threshold for a second pass (rf).
  const uint32_t c0     = PART == kFused || PART == kRank ? cd.cnt[qb] : 0u;
  const bool listed_all = c0 <= cd.cap;
  const int c           = static_cast<int>(min(c0, cd.cap));
  if constexpr (PART == kFused || PART == kRank) {
    if (!listed_all && rf.thr2 == nullptr) {
      give_up();
      return;
    }
    if (c == 0) {
      if (PART == kFused) {
        nothing();
      } else if (threadIdx.x == 0) {
        kept[qb] = 0;
      }
      return;
    }
    if (threadIdx.x == 0) { s_rows = 0, s_sure = 0, s_seen = 0, s_kept = 0; }
  }
  if constexpr (PART == kFused || PART == kScore) {
    const uint8_t* src = static_cast<const uint8_t*>(queries) + static_cast<size_t>(q) * qpitch;
    if constexpr (kBytes) {
      // the query's bytes, zero padded to whole 16-byte vectors, in the space of qd
      uint8_t* qbytes  = reinterpret_cast<uint8_t*>(qd);
      const int padded = (d + 15) / 16 * 16;
      for (int t = threadIdx.x; t < padded; t += blockDim.x) { qbytes[t] = t < d ? src[t] : 0; }
    } else {
      for (int t = threadIdx.x; t < d; t += blockDim.x) { qd[t] = Elems<T>::one(src, t); }
    }
  }
  if constexpr (!kBytes && PART != kRank) {  // |q|^2 in coordinate order, where the metric's scores have a use for it
    if (threadIdx.x == 0) { s_qq = METRIC == kL2 ? 0.0 : cd.qq[q]; }
  }
  __syncthreads();
  if constexpr (kBytes && PART != kRank) {
    if (threadIdx.x < 32) {  // |q|^2 as an integer: 255^2 * 4096 < 2^31
      const uint8_t* src = static_cast<const uint8_t*>(queries) + static_cast<size_t>(q) * qpitch;
      int a              = 0;
      for (int t = threadIdx.x; t < d; t += 32) {
        const int v = static_cast<int>(reinterpret_cast<const T*>(src)[t]);
        a += v * v;
      }
      a = __reduce_add_sync(0xffffffffu, a);
      if (threadIdx.x == 0) {
        s_qq_int = a;
        s_qq     = __ll2double_rn(static_cast<long long>(a));
      }
    }
    if (PART != kFused) { __syncthreads(); }
  }
  if constexpr (PART == kFused || PART == kRank) {
    // ---- values as unsigned keys in their order: of the rows that may be returned, and what every chain reaches (0: nothing)
    uint32_t* vkey    = PART == kRank ? reinterpret_cast<uint32_t*>(sh) : reinterpret_cast<uint32_t*>(sc);
    int32_t* vid      = reinterpret_cast<int32_t*>(vkey) + n2max;
    uint32_t* reached = PART == kRank ? vkey + 2 * n2max : reinterpret_cast<uint32_t*>(ids);
    auto id_of = [&](int64_t r) { return r < cd.n_rows ? __ldg(cd.perm + r) : cd.tail_id0 + static_cast<int32_t>(r - cd.n_rows); };
    auto key_of = [](int32_t product, int32_t e) {
      if constexpr (kBytes) {
        return static_cast<uint32_t>(product + e) ^ 0x80000000u;
      } else {
        const uint32_t f = __float_as_uint(__int_as_float(product) + __int_as_float(e));
        return f ^ ((f >> 31) ? 0xffffffffu : 0x80000000u);
      }
    };
    // Without a bitset the ids are looked up for the rows that are scored only: removed rows and padding have e = never.
    constexpr int32_t kNever = kBytes ? kNeverInit : static_cast<int32_t>(0xff800000u);
    const bool late          = adm.bits == nullptr && adm.row_labels == nullptr;
    int sure = 0, seen = 0;
    for (int i = threadIdx.x; i < c; i += blockDim.x) {
      const uint4 cv     = reinterpret_cast<const uint4*>(mine)[i];  // chain, mask, product
      const int32_t prod = static_cast<int32_t>(cv.z);
      uint32_t least     = 0xffffffffu;
      bool all           = true;
      for (uint32_t mask = cv.y; mask; mask &= mask - 1) {
        const int64_t r  = static_cast<int64_t>(cv.x) * kChainRows + __ffs(mask) - 1;
        const int32_t e  = r < cd.n_rows ? __ldg(cd.init + r) : r < cd.n_rows + cd.n_tail ? 0 : kNever;
        int32_t id       = static_cast<int32_t>(r);
        bool may         = e != kNever;
        if (may && !late) {
          id  = id_of(r);
          may = admitted(adm, q, id);
        }
        ++seen;
        if (may) {
          const uint32_t key = key_of(prod, e);
          const int at       = atomicAdd(&s_rows, 1);
          least              = min(least, key);
          if (at < n2max) { vkey[at] = key, vid[at] = id; }
        } else {
          all = false;
        }
      }
      reached[i] = all ? least : 0u;
      sure += all ? 1 : 0;
    }
    sure = __reduce_add_sync(0xffffffffu, sure);
    seen = __reduce_add_sync(0xffffffffu, seen);
    if ((threadIdx.x & 31) == 0) { atomicAdd(&s_sure, sure), atomicAdd(&s_seen, seen); }
    __syncthreads();
    const int rows  = min(s_rows, n2max);
    over            = !listed_all || s_rows > n2max;
    if (over && rf.thr2 == nullptr) {
      give_up();
      return;
    }
    uint32_t lowest = 1;
    if (s_sure >= k && s_rows > k) {
      lowest = block_kth_largest(reached, c, k, s_scratch);
      if constexpr (!kBytes) {
        const uint32_t f = lowest ^ ((lowest >> 31) ? 0x80000000u : 0xffffffffu);
        const float v    = __fadd_rd(__uint_as_float(f), -cd.shift[q]);
        const uint32_t g = __float_as_uint(v);
        lowest           = max(1u, g ^ ((g >> 31) ? 0xffffffffu : 0x80000000u));
      }
    }
    __syncthreads();  // the space of `reached` becomes the list of the rows to score
    for (int i = threadIdx.x; i < rows; i += blockDim.x) {
      if (vkey[i] >= lowest) {
        (PART == kRank ? far_ids : ids)[atomicAdd(&s_kept, 1)] = late ? id_of(vid[i]) : vid[i];
      }
    }
    __syncthreads();
    m = s_kept;
    if (threadIdx.x == 0 && stats) {
      atomicAdd(stats + 0, static_cast<unsigned long long>(s_seen));  // rows the screen kept
      atomicAdd(stats + 1, static_cast<unsigned long long>(m));       // exact scores computed
    }
    if (PART == kRank) {
      if (threadIdx.x == 0) { kept[qb] = m | (over ? 1 << 30 : 0); }
      return;
    }
  }
  if constexpr (kBytes) {
    unsigned long long* keys = reinterpret_cast<unsigned long long*>(sc);
    {
      // integer scores (below 2^31 in magnitude) and ids sort as one 64-bit key: (score + 2^31) << 32 | id
      constexpr int kGroups = 32 / kRowLanes;  // rows a warp's load covers
      const int sub         = threadIdx.x & (kRowLanes - 1);
      const int group       = (threadIdx.x >> 5) * kGroups + ((threadIdx.x & 31) / kRowLanes);
      const int n_groups    = (blockDim.x >> 5) * kGroups;
      for (int i0 = 0; i0 < m; i0 += n_groups * kRowUnroll) {  // the same trips for every lane of a warp
        int32_t row[kRowUnroll];
        long long v[kRowUnroll];
#pragma unroll
        for (int u = 0; u < kRowUnroll; ++u) {
          const int i = i0 + u * n_groups + group;
          row[u]      = i < m ? ids[i] : -1;
        }
        if (where) {  // `vectors` is not in id order: row `where[id]` of it holds the vector with that id
          int32_t at[kRowUnroll];
#pragma unroll
          for (int u = 0; u < kRowUnroll; ++u) { at[u] = row[u] >= 0 ? __ldg(where + row[u]) : -1; }
          int_row_scores<T, METRIC>(vectors, pitch, at, d, reinterpret_cast<const uint4*>(qd), s_qq_int, sub, v);
        } else {
          int_row_scores<T, METRIC>(vectors, pitch, row, d, reinterpret_cast<const uint4*>(qd), s_qq_int, sub, v);
        }
#pragma unroll
        for (int u = 0; u < kRowUnroll; ++u) {
          const int i = i0 + u * n_groups + group;
          if (sub == 0 && row[u] >= 0) {
            keys[i] = (static_cast<unsigned long long>(v[u] + 2147483648ll) << 32) | static_cast<uint32_t>(row[u]);
          }
        }
      }
    }
    if (PART == kScore) { return; }
    sort_keys(keys, m);
    if (over) {
      if (threadIdx.x == 0) {
        report_overflow<T, METRIC>(rf, q, qb, queries, qpitch, d, s_qq, k <= m ? __ll2double_rn(static_cast<long long>(keys[k - 1] >> 32) - 2147483648ll) : CUDART_INF, ovf_list, ovf_count);
      }
      return;
    }
    for (int t = threadIdx.x; t < k; t += blockDim.x) {
      const bool have                          = t < m;
      const unsigned long long key             = have ? keys[t] : 0ull;
      best_s[static_cast<size_t>(out) * k + t]   = have ? __ll2double_rn(static_cast<long long>(key >> 32) - 2147483648ll) : CUDART_INF;
      best_row[static_cast<size_t>(out) * k + t] = have ? static_cast<int32_t>(key & 0xffffffffull) : -1;
    }
  } else {
    {
      // Float rows: a thread sums its candidate's coordinates in order (the order of the fp64 reference loop), but the
      // rows come through shared memory: a warp fetches a 128-byte slab of 32 candidate rows with eight loads that each
      // cover four whole lines (eight lanes per row), parks it in its tile, and every lane then walks its own row's slab.
      // Per 512 bytes that is 4 + 4 + 4 memory wavefronts instead of the 32 of a warp whose lanes each load 16 bytes of
      // a different row.
      constexpr int V       = Elems<T>::kPerVec;  // coordinates per 16-byte piece
      const int lane        = threadIdx.x & 31, warp = threadIdx.x >> 5, n_warps = blockDim.x >> 5;
      const int n_pieces    = static_cast<int>((static_cast<size_t>(d) * sizeof(T) + 15) / 16);  // rows are zero padded to the pitch
      uint8_t* tile         = stage_of(PART == kFused ? static_cast<void*>(ids + n2max) : static_cast<void*>(qd + d)) + static_cast<size_t>(warp) * 32 * kStageStride;
      const int piece       = lane & 7, row_in_load = lane >> 3;
      for (int g = warp; g * 32 < m; g += n_warps) {
        const int i       = g * 32 + lane;
        const bool ok     = i < m;
        const int32_t row = ok ? ids[i] : -1;
        Acc<METRIC, 1, STORED_XX> acc;
        acc.clear();
        if constexpr (STORED_XX) {
          if (ok) { acc.xx = __ldg(sqnorm + row); }
        }
        int32_t from[8];  // the rows this lane fetches pieces of
#pragma unroll
        for (int j = 0; j < 8; ++j) { from[j] = __shfl_sync(0xffffffffu, row, 4 * j + row_in_load); }
        // The loads of the next slab are issued as soon as this slab's registers have been parked in the tile, so that
        // they are in flight while the lanes walk the tile (a warp alone then overlaps its memory latency with its sums).
        uint4 w[8];
        auto fetch = [&](int p0) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            w[j] = (from[j] >= 0 && p0 + piece < n_pieces)
                     ? __ldg(reinterpret_cast<const uint4*>(vectors + static_cast<size_t>(from[j]) * pitch) + p0 + piece)
                     : make_uint4(0, 0, 0, 0);
          }
        };
        fetch(0);
        for (int p0 = 0; p0 < n_pieces; p0 += 8) {
          __syncwarp();  // every lane is done with the slab before
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            *reinterpret_cast<uint4*>(tile + (4 * j + row_in_load) * kStageStride + piece * 16) = w[j];
          }
          __syncwarp();
          if (p0 + 8 < n_pieces) { fetch(p0 + 8); }
          if (ok) {
            const int np = min(8, n_pieces - p0);
            for (int p = 0; p < np; ++p) {
              const uint4 x4 = *reinterpret_cast<const uint4*>(tile + lane * kStageStride + p * 16);
              double x[V];
              Elems<T>::unpack_finite(x4, x);  // screened rows are finite
              const int t0 = (p0 + p) * V;
              if (t0 + V <= d) {
                // the query's doubles two at a time (t0 is a multiple of V, qd is 16-byte aligned): half the
                // shared-memory instructions of the walk
#pragma unroll
                for (int e = 0; e < V; e += 2) {
                  const double2 a = *reinterpret_cast<const double2*>(qd + t0 + e);
                  acc.add1(x[e], a.x);
                  acc.add1(x[e + 1], a.y);
                }
              } else {
                for (int e = 0; e < V && t0 + e < d; ++e) { acc.add(x[e], qd, d, t0 + e); }
              }
            }
          }
        }
        if (ok) { sc[i] = acc.result(0, s_qq); }
      }
    }
    if (PART == kScore) { return; }
    sort_pairs(sc, ids, m);
    if (over) {
      if (threadIdx.x == 0) { report_overflow<T, METRIC>(rf, q, qb, queries, qpitch, d, s_qq, k <= m ? sc[k - 1] : CUDART_INF, ovf_list, ovf_count); }
      return;
    }
    for (int t = threadIdx.x; t < k; t += blockDim.x) {
      const bool have                         = t < m;
      best_s[static_cast<size_t>(out) * k + t]   = have ? sc[t] : CUDART_INF;
      best_row[static_cast<size_t>(out) * k + t] = have ? ids[t] : -1;
    }
  }
}

// Sorts m entries in shared memory by (score, id): not inlined, it would cost the kernels registers that their usual path needs
// (sort_lists_kernel 64 -> 74 and a block per SM less, select_topk_kernel 2 - 4 % slower on plain scores).
constexpr int kSortCompares = 2048;
__device__ __noinline__ void sort_crowded(double* s, int32_t* id, int m)
{
  const int n2 = next_pow2(m);
  for (int i = m + threadIdx.x; i < n2; i += blockDim.x) { s[i] = CUDART_INF, id[i] = 0x7fffffff; }
  bitonic_sort(s, id, n2);
}

// Every thread of a block of NT: the m entries (score, id) that the threads hold (HELD each: entry threadIdx.x + i NT) in the
// order of (score, id): emit(place, score, id) for the first k places. The scores are spread over 4 NT intervals, the buckets
// are laid out one after the other in shared memory, and an entry's place is the beginning of its bucket plus the entries of
// the bucket that come before it. The intervals grow with the distance from the worst score (NT / 4 per octave, 16 octaves):
// the k best of a large set crowd at that end, the more so when a few are far better than the rest. A bitonic sort of 4096
// pairs moves 12 bytes an entry 78 times through shared memory, which bounds it: 217 us for 512 lists of 2400 entries; this one
// takes 44 us. An entry is compared with those of its interval, about 45 cycles each: where scores crowd (ties, or a spread
// of more than 16 octaves) so that a thread would make more than kSortCompares of them, the bitonic sort is what is left (a search
// of 200 queries that scores 5000 rows, k = 2048, all scores equal: 465 us by comparisons, 142 with this rule; all but five in one
// far cluster 470 and 155).
// Shared memory: s and id [next_pow2(m)] each | start [4 NT + 1], start 16-byte aligned.
template <int NT, int HELD, typename Emit>
__device__ void sort_block(const double (&x)[HELD], const int32_t (&xi)[HELD], int m, int k, double* s, int32_t* id, int32_t* start,
                           Emit&& emit)
{
  constexpr int B      = 4 * NT;
  constexpr int kShift = B == 4096 ? 15 : 17;  // of a float's bits: B / 16 intervals per octave
  static_assert(B == 4096 || B == 1024, "16 octaves");
  constexpr int W = NT / 32;
  __shared__ double s_lo[W], s_hi[W];
  __shared__ int s_sum[W], s_work[W];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double lo = CUDART_INF, hi = -CUDART_INF;
#pragma unroll
  for (int i = 0; i < HELD; ++i) {
    if (static_cast<int>(threadIdx.x) + i * NT < m) {
      lo = fmin(lo, x[i]);
      hi = fmax(hi, x[i]);
    }
  }
  for (int i = threadIdx.x; i <= B; i += NT) { start[i] = 0; }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  if (lane == 0) { s_lo[warp] = lo, s_hi[warp] = hi; }
  __syncthreads();
  lo = s_lo[lane & (W - 1)], hi = s_hi[lane & (W - 1)];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  // a larger score never has a smaller bucket: the difference, the product and the conversion round monotonically
  const double scale = hi > lo ? 1.0 / (hi - lo) : 0.0;
  auto bucket        = [&](double v) {
    const int far = static_cast<int>(__float_as_uint(__double2float_rn((hi - v) * scale)) >> kShift) - ((127 - 16) << (23 - kShift));
    return B - 1 - min(max(far, 0), B - 1);
  };
  int b[HELD], nth[HELD];
#pragma unroll
  for (int i = 0; i < HELD; ++i) {
    b[i] = -1;
    if (static_cast<int>(threadIdx.x) + i * NT < m) {
      b[i]   = bucket(x[i]);
      nth[i] = atomicAdd(&start[b[i]], 1);
    }
  }
  __syncthreads();
  // counts -> first places: four buckets per thread
  int4 c        = reinterpret_cast<int4*>(start)[threadIdx.x];
  const int sum = c.x + c.y + c.z + c.w;
  int incl      = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) { incl += v; }
  }
  const int work = __reduce_add_sync(0xffffffffu, c.x * c.x + c.y * c.y + c.z * c.z + c.w * c.w);  // at most m^2 in all
  if (lane == 31) { s_sum[warp] = incl, s_work[warp] = work; }
  __syncthreads();
  int before = incl - sum;
  for (int w = 0; w < warp; ++w) { before += s_sum[w]; }
  reinterpret_cast<int4*>(start)[threadIdx.x] = make_int4(before, before + c.x, before + c.x + c.y, before + c.x + c.y + c.z);
  if (threadIdx.x == 0) { start[B] = m; }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < HELD; ++i) {
    if (b[i] >= 0) {
      const int at = start[b[i]] + nth[i];
      s[at]        = x[i];
      id[at]       = xi[i];
    }
  }
  __syncthreads();
  int compares = 0;
  for (int w = 0; w < W; ++w) { compares += s_work[w]; }
  if (compares > kSortCompares * NT) {
    sort_crowded(s, id, m);
    for (int i = threadIdx.x; i < min(m, k); i += NT) { emit(i, s[i], id[i]); }
    return;
  }
#pragma unroll
  for (int i = 0; i < HELD; ++i) {
    if (b[i] >= 0) {
      const int first = start[b[i]], last = start[b[i] + 1];
      int place       = first;
      if (first < k) {
        for (int j = first; j < last; ++j) { place += pair_less(s[j], id[j], x[i], xi[i]) ? 1 : 0; }
        if (place < k) { emit(place, x[i], xi[i]); }
      }
    }
  }
}

// The third step of a split verification, block per query: its k best by (score, id).
template <typename T, int METRIC, int NT, int HELD>  // lists of at most NT HELD rows
__global__ void __launch_bounds__(NT, NT == 256 ? 4 : 1) sort_lists_kernel(const void* queries, size_t qpitch, int d, int q0, Candidates cd,
                                                                  int n2max, int k, double* best_s, int32_t* best_row,
                                                                  int32_t* ovf_list, unsigned int* ovf_count, Refine rf,
                                                                  const int32_t* kept)
{
  extern __shared__ double sh[];  // s [n2max] | id [n2max] | start [4 NT + 1]
  double* s           = sh;
  int32_t* id         = reinterpret_cast<int32_t*>(s + n2max);
  int32_t* start      = reinterpret_cast<int32_t*>(stage_of(id + n2max));  // 16-byte aligned
  const int qb        = blockIdx.x, q = q0 + qb;
  const int out       = cd.sel ? __ldg(cd.sel + q) : q;
  const int32_t w     = kept[qb];
  if (w < 0) { return; }  // given up
  const bool over     = (w >> 30) != 0;
  const int m         = w & 0x3fffffff;
  const double* far_s = reinterpret_cast<const double*>(cd.cand + static_cast<size_t>(qb) * cd.ld);
  double x[HELD];
  int32_t xi[HELD];
#pragma unroll
  for (int i = 0; i < HELD; ++i) {
    const int at = threadIdx.x + i * NT;
    x[i]         = CUDART_INF;
    xi[i]        = 0x7fffffff;
    if (at < m) {
      if constexpr (kByteRows<T>) {
        const unsigned long long key = reinterpret_cast<const unsigned long long*>(far_s)[at];
        x[i]                         = __ll2double_rn(static_cast<long long>(key >> 32) - 2147483648ll);
        xi[i]                        = static_cast<int32_t>(key & 0xffffffffull);
      } else {
        x[i]  = far_s[at];
        xi[i] = reinterpret_cast<const int32_t*>(far_s + n2max)[at];
      }
    }
  }
  sort_block<NT, HELD>(x, xi, m, k, s, id, start, [&](int place, double v, int32_t row) {
    if (!over) {
      best_s[static_cast<size_t>(out) * k + place]   = v;
      best_row[static_cast<size_t>(out) * k + place] = row;
    } else if (place == k - 1) {
      const double qq = METRIC == kL2 && !kByteRows<T> ? 0.0 : query_sqnorm<T>(cd, queries, qpitch, d, q);
      report_overflow<T, METRIC>(rf, q, qb, queries, qpitch, d, qq, v, ovf_list, ovf_count);
    }
  });
  if (over) {
    if (threadIdx.x == 0 && m < k) {
      report_overflow<T, METRIC>(rf, q, qb, queries, qpitch, d, 0.0, CUDART_INF, ovf_list, ovf_count);
    }
    return;
  }
  for (int t = m + threadIdx.x; t < k; t += NT) {
    best_s[static_cast<size_t>(out) * k + t]   = CUDART_INF;
    best_row[static_cast<size_t>(out) * k + t] = -1;
  }
}

// dst = src rounded to fp16, and *bad = 1 (in page-locked host memory) when a value is not finite in fp16; dst may be null:
// only the check. One pass over the values; eight per thread and turn where both arrays are 16-byte aligned.
template <typename T>
__device__ __forceinline__ float as_float(T v)
{
  if constexpr (std::is_same<T, __nv_bfloat16>::value) {
    return __bfloat162float(v);
  } else if constexpr (std::is_same<T, __half>::value) {
    return __half2float(v);
  } else {
    return v;
  }
}
template <typename T>
__global__ void to_half_kernel(const T* src, int64_t n, __half* dst, int aligned, volatile int* bad)
{
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  int64_t i            = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  bool out             = false;
  const int64_t n8     = aligned ? n / 8 : 0;
  constexpr int kLoads = sizeof(T) / 2;  // 16-byte loads for eight values
  for (int64_t g = i; g < n8; g += stride) {
    __align__(16) T v[8];
    __align__(16) __half h[8];
#pragma unroll
    for (int j = 0; j < kLoads; ++j) { reinterpret_cast<uint4*>(v)[j] = __ldg(reinterpret_cast<const uint4*>(src) + g * kLoads + j); }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      h[j] = __float2half_rn(as_float(v[j]));
      out |= __hisinf(h[j]) != 0 || __hisnan(h[j]);
    }
    if (dst) { reinterpret_cast<uint4*>(dst)[g] = *reinterpret_cast<const uint4*>(h); }
  }
  for (i += 8 * n8; i < n; i += stride) {
    const __half h = __float2half_rn(as_float(src[i]));
    out |= __hisinf(h) != 0 || __hisnan(h);
    if (dst) { dst[i] = h; }
  }
  if (out) { *bad = 1; }
}

// words[w] = bits 32 w .. 32 w + 31 of a mask of bytes (non-zero: set), one word per thread. Bound by reading the mask once:
// 1.2 M entries in 2.6 us (0.5 TB/s: one wave of blocks); as tensor operations ten launches, 40 us of them with their
// gaps and intermediate arrays of 64 bits per entry.
__global__ void pack_mask_kernel(const uint8_t* mask, int64_t n, uint32_t* words, int aligned)
{
  const int64_t w = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (w >= (n + 31) / 32) { return; }
  uint32_t out = 0;
  if (aligned && 32 * w + 32 <= n) {
    const uint4* p      = reinterpret_cast<const uint4*>(mask + 32 * w);
    const uint4 a       = __ldg(p), b = __ldg(p + 1);
    const uint32_t u[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      // bit 7 of every byte that is not zero, then the four bits side by side
      const uint32_t m = ((((u[i] & 0x7f7f7f7fu) + 0x7f7f7f7fu) | u[i]) & 0x80808080u) >> 7;
      out |= ((m * 0x01020408u) >> 24 & 0xfu) << (4 * i);
    }
  } else {
    const int m = static_cast<int>(min(static_cast<int64_t>(32), n - 32 * w));
    for (int i = 0; i < m; ++i) { out |= (mask[32 * w + i] != 0 ? 1u : 0u) << i; }
  }
  words[w] = out;
}

// out row i = in row sel[i] (or row i when sel is null), row_bytes of it, the rest of the out_pitch bytes zero; a negative
// sel[i] and rows [n, n_pad) give zero rows. 16-byte units when everything is 16-byte aligned.
__global__ void gather_rows_kernel(const uint8_t* in, size_t in_pitch, const int32_t* sel, int64_t n, uint8_t* out,
                                   size_t out_pitch, size_t row_bytes, int vec16)
{
  const int64_t row = blockIdx.x;
  int64_t from      = row < n ? (sel ? sel[row] : row) : -1;
  const uint8_t* src = from >= 0 ? in + static_cast<size_t>(from) * in_pitch : nullptr;
  uint8_t* dst       = out + static_cast<size_t>(row) * out_pitch;
  if (vec16) {
    const uint4 zero = make_uint4(0, 0, 0, 0);
    for (size_t b = threadIdx.x; b < out_pitch / 16; b += blockDim.x) {
      reinterpret_cast<uint4*>(dst)[b] = (src && b < row_bytes / 16) ? reinterpret_cast<const uint4*>(src)[b] : zero;
    }
  } else {
    for (size_t b = threadIdx.x; b < out_pitch; b += blockDim.x) { dst[b] = (src && b < row_bytes) ? src[b] : 0; }
  }
}

// Label layout of the partition entries: entry p (id part_ids[p], label number i found by its offset) goes to row
// lrow0[i] + (p - off[i]) of the label-ordered copy. Writes lperm [lrow] = id, linv [id] = lrow, lsrc [lrow] = the
// sorted row the codes are copied from, linit [lrow] = e of that row.
__global__ void label_rows_kernel(const int32_t* part_ids, int64_t n, const int64_t* off, const int64_t* lrow0, int n_labels,
                                  const int32_t* inv, const int32_t* init, int32_t* lperm, int32_t* linv, int32_t* lsrc,
                                  int32_t* linit)
{
  const int64_t p = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (p >= n) { return; }
  int lo = 0, hi = n_labels - 1;  // last label whose first entry is <= p
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (off[mid] <= p) {
      lo = mid;
    } else {
      hi = mid - 1;
    }
  }
  const int32_t id   = part_ids[p];
  const int64_t lrow = lrow0[lo] + (p - off[lo]);
  const int32_t srow = inv[id];
  lperm[lrow] = id;
  linv[id]    = static_cast<int32_t>(lrow);
  lsrc[lrow]  = srow;
  linit[lrow] = init[srow];
}

// best lists of the compact queries 0 .. n - 1 -> rows sel[i] of the call's lists
__global__ void scatter_best_kernel(const double* s2, const int32_t* row2, const int32_t* sel, int k, double* best_s,
                                    int32_t* best_row)
{
  if (sel[blockIdx.x] < 0) { return; }
  const size_t src = static_cast<size_t>(blockIdx.x) * k, dst = static_cast<size_t>(sel[blockIdx.x]) * k;
  for (int t = threadIdx.x; t < k; t += blockDim.x) {
    best_s[dst + t]   = s2[src + t];
    best_row[dst + t] = row2[src + t];
  }
}

// list[i] = sel[list[i]]: compact query numbers back to the numbers of the call
__global__ void compose_kernel(int32_t* list, const unsigned int* n, const int32_t* sel)
{
  const unsigned int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < *n) { list[i] = sel[list[i]]; }
}

// ------------------------------------------------------------------------------------------- dense path
constexpr int kDenseQ = 4;  // queries per block that share one walk over a stored row
constexpr size_t kDenseMost = kMaxSmem - 256;  // dynamic shared memory of a block of them, beside their own variables

template <typename T, int METRIC>
__global__ void dense_scores_kernel(const uint8_t* vectors, size_t pitch, int d, int64_t n, const void* queries,
                                    size_t qpitch, const int32_t* qsel, int q0, int nqb, Admit adm, double* out, int64_t ld)
{
  extern __shared__ double sh[];
  __shared__ double s_qq[kDenseQ];
  __shared__ int64_t s_qidx[kDenseQ];
  const int b0 = blockIdx.y * kDenseQ;
  const int nb = min(kDenseQ, nqb - b0);
  if (threadIdx.x < kDenseQ) {
    const int b = min(static_cast<int>(threadIdx.x), nb - 1);
    s_qidx[threadIdx.x] = qsel ? qsel[b0 + b] : q0 + b0 + b;
  }
  __syncthreads();
  load_queries<T>(queries, qpitch, s_qidx, kDenseQ, d, sh, d, s_qq);
  const int64_t row = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (row >= n) { return; }
  Acc<METRIC, kDenseQ> acc;
  acc.clear();
  scan_row<T, METRIC, kDenseQ>(vectors + static_cast<size_t>(row) * pitch, d, sh, d, acc);
#pragma unroll
  for (int b = 0; b < kDenseQ; ++b) {
    if (b < nb) {
      const bool ok = admitted(adm, s_qidx[b], row);
      out[static_cast<int64_t>(b0 + b) * ld + row] = ok ? acc.result(b, s_qq[b]) : CUDART_INF;
    }
  }
}

// Dense scores of label groups in one launch. Group g pairs the queries order[q_begin .. q_begin + nq) (all of one
// label) with the columns of that label: the n_part ids part_ids[part_off ..] of the label partition, then the rows
// tail0 .. tail0 + n_tail - 1 added after the partition was made (`adm` keeps those of the query's label). Blocks
// blk_begin[g] .. blk_begin[g + 1] - 1 belong to group g: quads of queries (slow) by chunks of 256 columns (fast).
template <typename T, int METRIC>
__global__ void dense_scores_grouped_kernel(const uint8_t* vectors, size_t pitch, int d, const void* queries, size_t qpitch,
                                            const int32_t* order, const LabelGroup* groups, int n_groups,
                                            const int32_t* part_ids, int64_t tail0, int64_t n_tail, Admit adm, double* out)
{
  extern __shared__ double sh[];
  __shared__ double s_qq[kDenseQ];
  __shared__ int64_t s_qidx[kDenseQ];
  int lo = 0, hi = n_groups - 1;  // last group whose first block is <= blockIdx.x
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (groups[mid].blk_begin <= static_cast<int64_t>(blockIdx.x)) {
      lo = mid;
    } else {
      hi = mid - 1;
    }
  }
  const LabelGroup g    = groups[lo];
  const int64_t n_cols  = g.n_part + n_tail;
  const int64_t chunks  = (n_cols + blockDim.x - 1) / blockDim.x;
  const int64_t local   = static_cast<int64_t>(blockIdx.x) - g.blk_begin;
  const int b0          = static_cast<int>(local / chunks) * kDenseQ;
  const int64_t col     = (local % chunks) * blockDim.x + threadIdx.x;
  const int nb          = min(kDenseQ, g.nq - b0);
  if (threadIdx.x < kDenseQ) {
    const int b         = min(static_cast<int>(threadIdx.x), nb - 1);
    s_qidx[threadIdx.x] = order[g.q_begin + b0 + b];
  }
  __syncthreads();
  load_queries<T>(queries, qpitch, s_qidx, kDenseQ, d, sh, d, s_qq);
  if (col >= n_cols) { return; }
  const int64_t row = col < g.n_part ? part_ids[g.part_off + col] : tail0 + (col - g.n_part);
  Acc<METRIC, kDenseQ> acc;
  acc.clear();
  scan_row<T, METRIC, kDenseQ>(vectors + static_cast<size_t>(row) * pitch, d, sh, d, acc);
#pragma unroll
  for (int b = 0; b < kDenseQ; ++b) {
    if (b < nb) {
      const bool ok = admitted(adm, s_qidx[b], row);
      out[g.score_off + static_cast<int64_t>(b0 + b) * g.ld + col] = ok ? acc.result(b, s_qq[b]) : CUDART_INF;
    }
  }
}

// Columns of a label group's score row -> ids, for the k winners of every query of the group (see above).
__global__ void group_columns_to_ids_kernel(int32_t* best_row, int k, const int32_t* order, const LabelGroup* groups,
                                            const int32_t* part_ids, int64_t tail0)
{
  const LabelGroup g = groups[blockIdx.x];
  for (int i = threadIdx.x; i < g.nq * k; i += blockDim.x) {
    const size_t o    = static_cast<size_t>(order[g.q_begin + i / k]) * k + (i % k);
    const int32_t col = best_row[o];
    if (col >= 0) { best_row[o] = col < g.n_part ? part_ids[g.part_off + col] : static_cast<int32_t>(tail0 + (col - g.n_part)); }
  }
}

// Block per query: the k smallest (score, row) of a row of scores (+inf and NaN: rows that do not count), sorted and written.
// Bound by reading the row: once for its smallest and largest key, once for a histogram of 2048 intervals between them, once to
// take the winners and the rows of the interval that holds the k-th, whose last places are given by counting. (A walk over fixed
// 8-bit digits reads the row nine times, and its counters wait for one another: in the upper digits the scores of a row
// are alike. 352 rows of 14 775 scores on average, k = 2048: 368 us; this one 99 us.) When the interval holds more than kPool rows,
// or so many that counting their places takes longer than reading the row once more (200 rows of 5000 scores over 15 orders of
// magnitude, k = 2048: 405 us a call with up to kPool in any case, 163 with both rules), it is divided again; scores that are all
// equal go to the smallest rows.
// Shared memory: sel_s [kk] doubles | sel_id [kk] int32 | pool_s [kPool] doubles | pool_id [kPool] int32 | bins, and after them
// the sort's buckets; kk = k rounded up to a multiple of 4.
// With `row_off` the score rows are ragged: row blockIdx.x starts at scores + row_off[blockIdx.x] and has row_n[] columns.
constexpr int kPool = 1024, kBins = 2048;
template <int NT>
constexpr size_t select_smem(int k)
{
  return 12 * (static_cast<size_t>((k + 3) / 4 * 4) + kPool) + 4 * static_cast<size_t>(kBins > 4 * NT + 4 ? kBins : 4 * NT + 4);
}
template <int NT>
__global__ void __launch_bounds__(NT) select_topk_kernel(const double* scores, int64_t ld, int64_t n_all, int k, const int32_t* qsel, int q0,
                                                         double* best_s, int32_t* best_row, int64_t chunk, double* part_s,
                                                         int32_t* part_row, const int64_t* row_off, const int32_t* row_n)
{
  using u64 = unsigned long long;
  constexpr int W = NT / 32, kHeld = 2048 / NT;
  extern __shared__ double sh[];
  __shared__ u64 s_min[W], s_max[W];
  __shared__ int s_cnt[W], s_less, s_pool, s_bin, s_before, s_in_bin, s_eq;
  const int kk    = (k + 3) / 4 * 4;
  double* sel_s   = sh;
  double* pool_s  = sel_s + kk;
  int32_t* sel_id = reinterpret_cast<int32_t*>(pool_s + kPool);
  int32_t* pool_id = sel_id + kk;
  int32_t* bins   = pool_id + kPool;  // 16-byte aligned: everything before is a multiple of 16 bytes
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // blockIdx.y selects a chunk of columns [col0, col0 + n); with several chunks the winners go to part_* and are merged
  const int64_t col0 = static_cast<int64_t>(blockIdx.y) * chunk;
  if (row_off) { n_all = row_n[blockIdx.x]; }
  const int64_t n    = max(static_cast<int64_t>(0), min(chunk, n_all - col0));
  const double* row  = scores + (row_off ? row_off[blockIdx.x] : static_cast<int64_t>(blockIdx.x) * ld) + col0;
  const int64_t qout = qsel ? qsel[blockIdx.x] : q0 + static_cast<int>(blockIdx.x);

  u64 lo = ~0ull, hi = 0;
  int counted = 0;
#pragma unroll 4
  for (int64_t i = threadIdx.x; i < n; i += NT) {
    const double v = row[i];
    if (v < CUDART_INF) {
      const u64 key = ordered_key(v);
      lo = key < lo ? key : lo, hi = key > hi ? key : hi;
      ++counted;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const u64 a = __shfl_xor_sync(0xffffffffu, lo, o), b = __shfl_xor_sync(0xffffffffu, hi, o);
    lo = a < lo ? a : lo, hi = b > hi ? b : hi;
  }
  counted = __reduce_add_sync(0xffffffffu, counted);
  if (lane == 0) { s_min[warp] = lo, s_max[warp] = hi, s_cnt[warp] = counted; }
  if (threadIdx.x == 0) { s_less = 0, s_pool = 0, s_eq = 0; }
  __syncthreads();
  counted = 0;
  for (int w = 0; w < W; ++w) {
    lo = s_min[w] < lo ? s_min[w] : lo, hi = s_max[w] > hi ? s_max[w] : hi;
    counted += s_cnt[w];
  }
  const int want = min(k, counted);
  if (want > 0) {
    // the interval [prefix << shift, (prefix + 1) << shift) of key - lo that holds the last winner
    int above = 64 - __clzll(static_cast<long long>(hi - lo));  // bits of key - lo above which nothing differs
    int shift = max(above - 11, 0), in_bin = 0, remaining = want;
    bool pooled = false;
    u64 prefix = 0;
    while (true) {
      const u64 inside = (1ull << (above - shift)) - 1;  // 11 bits, or what is left
      for (int i = threadIdx.x; i < kBins; i += NT) { bins[i] = 0; }
      __syncthreads();
#pragma unroll 4
      for (int64_t i = threadIdx.x; i < n; i += NT) {
        const double v = row[i];
        if (v < CUDART_INF) {
          const u64 d = ordered_key(v) - lo;
          if (above == 64 || (d >> above) == prefix) { atomicAdd(&bins[(d >> shift) & inside], 1); }
        }
      }
      __syncthreads();
      // bins per thread in order, their running sum: the bin where it reaches `remaining`
      constexpr int P = kBins / NT;
      int c[P], sum = 0;
#pragma unroll
      for (int i = 0; i < P; ++i) { c[i] = bins[threadIdx.x * P + i], sum += c[i]; }
      int incl = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) { incl += v; }
      }
      if (lane == 31) { s_cnt[warp] = incl; }
      __syncthreads();
      int before = incl - sum;
      for (int w = 0; w < warp; ++w) { before += s_cnt[w]; }
      if (before < remaining && before + sum >= remaining) {
        bool found = false;
#pragma unroll
        for (int i = 0; i < P; ++i) {
          if (!found && before + c[i] >= remaining) {
            s_bin = threadIdx.x * P + i, s_before = before, s_in_bin = c[i];
            found = true;
          }
          before += c[i];
        }
      }
      __syncthreads();
      prefix = (prefix << (above - shift)) + static_cast<u64>(s_bin);
      remaining -= s_before;
      in_bin = s_in_bin;
      pooled = in_bin <= kPool && static_cast<int64_t>(in_bin) * in_bin <= 4 * n + 64 * NT;
      if (pooled || shift == 0) { break; }
      above = shift;
      shift = max(shift - 11, 0);
    }
    const int n_less = want - remaining;
    for (int64_t i0 = 0; i0 < n; i0 += NT) {
      const int64_t i = i0 + threadIdx.x;
      const double v  = i < n ? row[i] : CUDART_INF;
      const u64 d     = v < CUDART_INF ? (ordered_key(v) - lo) >> shift : ~0ull;
      const bool less = v < CUDART_INF && d < prefix, eq = v < CUDART_INF && d == prefix;
      const uint32_t bl = __ballot_sync(0xffffffffu, less), be = __ballot_sync(0xffffffffu, eq);
      const uint32_t lt = (1u << lane) - 1u;
      if (bl) {
        int at = 0;
        if (lane == 0) { at = atomicAdd(&s_less, __popc(bl)); }
        at = __shfl_sync(0xffffffffu, at, 0) + __popc(bl & lt);
        if (less) { sel_s[at] = v, sel_id[at] = static_cast<int32_t>(col0 + i); }
      }
      if (pooled) {
        if (be) {
          int at = 0;
          if (lane == 0) { at = atomicAdd(&s_pool, __popc(be)); }
          at = __shfl_sync(0xffffffffu, at, 0) + __popc(be & lt);
          if (eq) { pool_s[at] = v, pool_id[at] = static_cast<int32_t>(col0 + i); }
        }
      } else if (__syncthreads_or(eq)) {  // equal scores: the smallest rows, in the order of the row
        if (lane == 0) { s_cnt[warp] = __popc(be); }
        __syncthreads();
        int at = s_eq + __popc(be & lt), total = 0;
        for (int w = 0; w < W; ++w) {
          at += w < warp ? s_cnt[w] : 0;
          total += s_cnt[w];
        }
        if (eq && at < remaining) { sel_s[n_less + at] = v, sel_id[n_less + at] = static_cast<int32_t>(col0 + i); }
        __syncthreads();
        if (threadIdx.x == 0) { s_eq += total; }
        __syncthreads();
      }
    }
    __syncthreads();
    if (pooled) {
      for (int i = threadIdx.x; i < in_bin; i += NT) {
        const double v   = pool_s[i];
        const int32_t vi = pool_id[i];
        int place        = 0;
        for (int j = 0; j < in_bin; ++j) { place += pair_less(pool_s[j], pool_id[j], v, vi) ? 1 : 0; }
        if (place < remaining) { sel_s[n_less + place] = v, sel_id[n_less + place] = vi; }
      }
      __syncthreads();
    }
  }
  double x[kHeld];
  int32_t xi[kHeld];
#pragma unroll
  for (int i = 0; i < kHeld; ++i) {
    const int at = threadIdx.x + i * NT;
    x[i]         = at < want ? sel_s[at] : CUDART_INF;
    xi[i]        = at < want ? sel_id[at] : 0;
  }
  const size_t out = part_s ? (static_cast<size_t>(blockIdx.x) * gridDim.y + blockIdx.y) * k : static_cast<size_t>(qout) * k;
  double* out_s    = part_s ? part_s : best_s;
  int32_t* out_row = part_s ? part_row : best_row;
  __syncthreads();
  sort_block<NT, kHeld>(x, xi, want, k, sel_s, sel_id, bins, [&](int place, double v, int32_t r) {
    out_s[out + place]   = v;
    out_row[out + place] = r;
  });
  for (int t = want + threadIdx.x; t < k; t += NT) {
    out_s[out + t]   = CUDART_INF;
    out_row[out + t] = part_s ? 0x7fffffff : -1;
  }
}

// Block per query: the k best of `parts` partial lists of k (score, row) pairs each, by (score, row).
// Shared memory: s [n2] doubles | row [n2] int32.
__global__ void merge_partials_kernel(const double* part_s, const int32_t* part_row, int parts, int k, int n2,
                                      const int32_t* qsel, int q0, double* best_s, int32_t* best_row)
{
  extern __shared__ double sh[];
  double* s    = sh;
  int32_t* row = reinterpret_cast<int32_t*>(sh + n2);
  const int m  = parts * k;
  for (int i = threadIdx.x; i < n2; i += blockDim.x) {
    s[i]   = i < m ? part_s[static_cast<size_t>(blockIdx.x) * m + i] : CUDART_INF;
    row[i] = i < m ? part_row[static_cast<size_t>(blockIdx.x) * m + i] : 0x7fffffff;
  }
  bitonic_sort(s, row, n2);
  const int64_t qout = qsel ? qsel[blockIdx.x] : q0 + static_cast<int>(blockIdx.x);
  for (int t = threadIdx.x; t < k; t += blockDim.x) {
    const bool have                            = s[t] < CUDART_INF;
    best_s[static_cast<size_t>(qout) * k + t]   = have ? s[t] : CUDART_INF;
    best_row[static_cast<size_t>(qout) * k + t] = have ? row[t] : -1;
  }
}

// ------------------------------------------------------------------------------------------- output
// Block per query. Distances as `finish` of the reference returns them (cpp/src/neighbors/certex/certex.cu:224-250).
template <typename T>
__global__ void finish_kernel(const double* best_s, const int32_t* best_row, const int64_t* best_id, int64_t id_base,
                              const void* queries, size_t qpitch, int d, int metric, int k, int64_t* neighbors,
                              float* distances, double* scores_out)
{
  __shared__ double s_qq;
  const int q = blockIdx.x;
  if (metric == kIP) {
    if (threadIdx.x == 0) {
      const uint8_t* src = static_cast<const uint8_t*>(queries) + static_cast<size_t>(q) * qpitch;
      double a           = 0;
      for (int t = 0; t < d; ++t) {
        const double v = Elems<T>::one(src, t);
        a              = __dadd_rn(a, __dmul_rn(v, v));
      }
      s_qq = a;
    }
    __syncthreads();
  }
  for (int t = threadIdx.x; t < k; t += blockDim.x) {
    const size_t o   = static_cast<size_t>(q) * k + t;
    const double s   = best_s[o];
    int64_t id       = -1;
    if (best_row) {
      if (best_row[o] >= 0) { id = id_base + best_row[o]; }
    } else {
      id = best_id[o];
    }
    float dist;
    if (id < 0) {
      dist = metric == kIP ? -CUDART_INF_F : CUDART_INF_F;
    } else if (metric == kL2) {
      dist = static_cast<float>(s);
    } else if (metric == kIP) {
      dist = static_cast<float>((s_qq - s) / 2);
    } else {
      dist = static_cast<float>(s / 2);
    }
    neighbors[o] = id;
    distances[o] = dist;
    if (scores_out) { scores_out[o] = id < 0 ? CUDART_INF : s; }
  }
}

// Block per query; shared memory: s [n2] doubles | id [n2] int64.
__global__ void search_status_kernel(const unsigned int* count, const unsigned int* q_ovf, unsigned long long* status)
{
  *status = (count[0] != 0 ? 1ull : 0ull) | (count[1] != 0 ? 2ull : 0ull) | (*q_ovf != 0 ? 4ull : 0ull);
}

__global__ void merge_kernel(const double* in_s, const int64_t* in_id, int parts, int nq, int k, int n2, double* out_s,
                             int64_t* out_id, int64_t part_stride)
{
  extern __shared__ double sh[];
  double* s   = sh;
  int64_t* id = reinterpret_cast<int64_t*>(sh + n2);
  const int q = blockIdx.x;
  const int m = parts * k;
  for (int i = threadIdx.x; i < n2; i += blockDim.x) {
    double v   = CUDART_INF;
    int64_t ii = 0x7fffffffffffffffll;
    if (i < m) {
      const size_t o = static_cast<size_t>(i / k) * part_stride + static_cast<size_t>(q) * k + (i % k);
      if (in_id[o] >= 0) {
        v  = in_s[o];
        ii = in_id[o];
      }
    }
    s[i]  = v;
    id[i] = ii;
  }
  bitonic_sort(s, id, n2);
  for (int t = threadIdx.x; t < k; t += blockDim.x) {
    const bool have                      = id[t] != 0x7fffffffffffffffll;
    out_s[static_cast<size_t>(q) * k + t]  = have ? s[t] : CUDART_INF;
    out_id[static_cast<size_t>(q) * k + t] = have ? id[t] : -1;
  }
}

// The same merge with a warp per query, for parts * k <= kMergeSmallMax candidates: every candidate's place is the number
// of candidates that come before it by (score, id); the first k are written. Shared memory: m doubles + m int64 per warp.
constexpr int kMergeSmallMax = 256;
__global__ void merge_small_kernel(const double* in_s, const int64_t* in_id, int parts, int nq, int k, double* out_s,
                                   int64_t* out_id, int64_t part_stride)
{
  extern __shared__ double merge_smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int q    = blockIdx.x * warps + warp;
  if (q >= nq) { return; }  // warps are independent: no block-wide barrier below
  const int m = parts * k;
  double* s   = merge_smem + static_cast<size_t>(warp) * m;
  int64_t* id = reinterpret_cast<int64_t*>(merge_smem + static_cast<size_t>(warps) * m) + static_cast<size_t>(warp) * m;
  for (int i = lane; i < m; i += 32) {
    const size_t o = static_cast<size_t>(i / k) * part_stride + static_cast<size_t>(q) * k + (i % k);
    const int64_t ii = in_id[o];
    s[i]  = ii >= 0 ? in_s[o] : CUDART_INF;
    id[i] = ii >= 0 ? ii : 0x7fffffffffffffffll;
  }
  __syncwarp();
  for (int i = lane; i < m; i += 32) {
    const double x   = s[i];
    const int64_t xi = id[i];
    int place        = 0;
    for (int j = 0; j < m; ++j) {
      const double y   = s[j];
      const int64_t yi = id[j];
      place += (y < x || (y == x && (yi < xi || (yi == xi && j < i)))) ? 1 : 0;
    }
    if (place < k) {
      const bool have                           = xi != 0x7fffffffffffffffll;
      out_s[static_cast<size_t>(q) * k + place]  = have ? x : CUDART_INF;
      out_id[static_cast<size_t>(q) * k + place] = have ? xi : -1;
    }
  }
}

template <typename F>
void by_dtype(int dtype, F&& f)
{
  switch (dtype) {
    case kF32: f(float{}); break;
    case kF16: f(__half{}); break;
    case kI8: f(int8_t{}); break;
    default: f(uint8_t{}); break;
  }
}

/// Opts in to the shared memory of a launch. The limit belongs to the function on its device, not to the calling thread: it is
/// set to `most`, the largest that any launch of the kernel takes, so that a thread with a small call cannot lower it
/// between another thread's call of this function and its launch. (Setting it each time serves every device and context.)
template <typename Kernel>
void allow_smem(Kernel kernel, size_t bytes, size_t most)
{
  // the 48 KB that need no opt-in include the kernel's static shared memory: leave room for it
  if (bytes > 32 * 1024) {
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(std::max(bytes, most)));
  }
}

}  // namespace

// ------------------------------------------------------------------------------------------- launchers
void launch_row_init(const void* vectors, size_t pitch, int dtype, int d, int metric, const uint8_t* removed,
                     int64_t row0, int64_t n, int64_t n_pad, int32_t* init, cudaStream_t s)
{
  const int64_t rows = n_pad - row0;
  if (rows <= 0) { return; }
  const int64_t threads = rows * 8;
  const int block       = 256;
  const auto grid       = static_cast<unsigned>((threads + block - 1) / block);
  if (dtype == kI8) {
    row_init_kernel<int8_t><<<grid, block, 0, s>>>(static_cast<const uint8_t*>(vectors), pitch, d, metric, removed, row0, n, n_pad, init);
  } else {
    row_init_kernel<uint8_t><<<grid, block, 0, s>>>(static_cast<const uint8_t*>(vectors), pitch, d, metric, removed, row0, n, n_pad, init);
  }
}

void launch_gather_init(const int32_t* init, int64_t stride, int64_t n_tiles, int32_t* out, cudaStream_t s,
                        const uint32_t* bits, const int32_t* perm, int32_t never)
{
  if (n_tiles <= 0) { return; }
  gather_init_kernel<<<static_cast<unsigned>(n_tiles), kBaseTile, 0, s>>>(init, stride, n_tiles, out, bits, perm, never);
}

void launch_gather_chain_min(const int32_t* init, int64_t stride_w, int64_t stride_i, int64_t stride_t, int64_t n_tiles,
                             int32_t* out, bool is_float, cudaStream_t s)
{
  if (n_tiles <= 0) { return; }
  const int64_t n = n_tiles * (kBaseTile / kChainRows);
  gather_chain_min_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, s>>>(init, stride_w, stride_i, stride_t, n_tiles, out,
                                                                                 is_float ? 1 : 0);
}

void launch_candidate_rows(const Candidate* cand, const uint32_t* cnt, uint32_t cap, int nq, int64_t n_rows, uint32_t* row_cnt,
                           int32_t* rows, uint32_t row_cap, cudaStream_t s)
{
  if (nq > 0) { candidate_rows_kernel<<<nq, 128, 0, s>>>(cand, cnt, cap, n_rows, row_cnt, rows, row_cap); }
}

void launch_tail(const TailRows& t, const uint8_t* q_codes, const int32_t* thr, const int32_t* label, const int32_t* slot0,
                 const int32_t* n_slots, int n_runs, Candidate* cand, uint32_t* cnt, uint32_t cap, int ld, cudaStream_t s)
{
  if (t.n_tail <= 0 || n_runs <= 0) { return; }
  const auto grid = static_cast<unsigned>(std::min<int64_t>((static_cast<int64_t>(t.n_tail) + 7) / 8, 148 * 8));
  auto kernel     = t.kind == 2 ? tail_kernel<2> : t.kind == 1 ? tail_kernel<1> : tail_kernel<0>;
  kernel<<<grid, 256, 0, s>>>(t, q_codes, thr, label, slot0, n_slots, n_runs, cand, cnt, cap, ld);
}

void launch_chain_max(const int32_t* init, int64_t c0, int64_t n, int32_t* cmax, bool is_float, cudaStream_t s)
{
  if (n <= 0) { return; }
  const auto grid = static_cast<unsigned>((n + 255) / 256);
  if (is_float) {
    chain_max_f32_kernel<<<grid, 256, 0, s>>>(reinterpret_cast<const float*>(init), c0, n, reinterpret_cast<float*>(cmax));
  } else {
    chain_max_kernel<<<grid, 256, 0, s>>>(init, c0, n, cmax);
  }
}

void launch_encode_f16_rows(const void* vectors, size_t pitch, int dtype, int d, int metric, int64_t n, void* codes,
                            size_t code_pitch, float* e, unsigned int* maxima, cudaStream_t s)
{
  if (n <= 0) { return; }
  by_dtype(dtype, [&](auto tag) {
    using T = decltype(tag);
    if constexpr (!kByteRows<T>) {
      const bool wide = d > 32 * Elems<T>::kPerVec;
      auto go = [&](auto kernel, int rows) {
        const int64_t blocks = std::min<int64_t>((n + rows - 1) / rows, kEncodeBlocks);
        kernel<<<static_cast<unsigned>(blocks), kEncodeThreads, 0, s>>>(static_cast<const uint8_t*>(vectors), pitch, d, metric, n,
                                                                        static_cast<uint8_t*>(codes), code_pitch, e, maxima);
      };
      if (wide) {
        go(encode_f16_rows_kernel<T, 32>, kEncodeThreads / 32);
      } else {
        go(encode_f16_rows_kernel<T, 8>, kEncodeThreads / 8);
      }
    }
  });
}

void launch_encode_f16_queries(const void* queries, size_t qpitch, int dtype, int d, int64_t nq, int64_t nq_pad, void* codes,
                               size_t code_pitch, float n1max, float n2max, float emax, float* shift,
                               unsigned int* overflow, cudaStream_t s)
{
  if (nq <= 0) { return; }
  const auto grid = static_cast<unsigned>((nq_pad * 32 + 255) / 256);
  if (dtype == kF32) {
    encode_f16_queries_kernel<float><<<grid, 256, 0, s>>>(static_cast<const uint8_t*>(queries), qpitch, d, nq, nq_pad,
                                                          static_cast<uint8_t*>(codes), code_pitch, n1max, n2max, emax, shift, overflow);
  } else {
    encode_f16_queries_kernel<__half><<<grid, 256, 0, s>>>(static_cast<const uint8_t*>(queries), qpitch, d, nq, nq_pad,
                                                           static_cast<uint8_t*>(codes), code_pitch, n1max, n2max, emax, shift, overflow);
  }
}

void launch_query_sqnorms(const void* queries, size_t qpitch, int dtype, int d, int64_t nq, double* qq, cudaStream_t s)
{
  if (nq <= 0) { return; }
  const auto grid = static_cast<unsigned>((nq + 31) / 32);
  if (dtype == kF32) {
    query_sqnorm_kernel<float><<<grid, 32, 0, s>>>(static_cast<const uint8_t*>(queries), qpitch, d, nq, qq);
  } else {
    query_sqnorm_kernel<__half><<<grid, 32, 0, s>>>(static_cast<const uint8_t*>(queries), qpitch, d, nq, qq);
  }
}

void launch_finish_thr_f16(int32_t* thr, const float* shift, int nq, int step, cudaStream_t s, int per)
{
  if (nq <= 0) { return; }
  finish_thr_f16_kernel<<<(nq + 255) / 256, 256, 0, s>>>(thr, shift, nq, step, per);
}

void launch_union_kth(const int32_t* parts, int n_parts, int nq, int k, int32_t* scratch, int32_t* thr, cudaStream_t s)
{
  if (nq <= 0) { return; }
  const int m       = n_parts * k;
  if (m <= kUnionMax) {  // a warp per query ranks the values by counting
    const int warps = 4;
    union_kth_kernel<<<(nq + warps - 1) / warps, warps * 32, static_cast<size_t>(warps) * m * 4, s>>>(parts, n_parts, nq, k, thr);
    return;
  }
  const int64_t ld  = (m + 7) / 8 * 8;
  const int64_t tot = static_cast<int64_t>(nq) * m;
  union_rows_kernel<<<static_cast<unsigned>((tot + 255) / 256), 256, 0, s>>>(parts, n_parts, nq, k, scratch, ld);
  launch_kth_largest(scratch, ld, m, k, nq, thr, s);
}

void launch_fill_i32(int32_t* p, int64_t n, int32_t v, cudaStream_t s)
{
  if (n <= 0) { return; }
  fill_i32_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, s>>>(p, n, v);
}

void launch_mask_removed(int32_t* e, const uint8_t* removed, int64_t n, bool is_float, cudaStream_t s)
{
  if (n <= 0) { return; }
  const int32_t never = is_float ? static_cast<int32_t>(0xff800000u) : kNeverInit;
  mask_removed_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, s>>>(e, removed, n, never);
}

size_t sort_batch_temp_bytes(int64_t n)
{
  size_t bytes = 0;
  cub::DeviceRadixSort::SortPairs(nullptr, bytes, static_cast<const uint32_t*>(nullptr), static_cast<uint32_t*>(nullptr),
                                  static_cast<const int32_t*>(nullptr), static_cast<int32_t*>(nullptr), n);
  return bytes;
}

void launch_sort_batch(const int32_t* e, int64_t n, int32_t id0, int64_t row0, const void* src, int64_t src_id0, size_t pitch,
                       int metric, bool is_float, uint32_t* keys_in, uint32_t* keys_out, int32_t* ids_in, int32_t* ids_out,
                       void* temp, size_t temp_bytes, void* codes, int32_t* perm, int32_t* inv, int32_t* init, cudaStream_t s)
{
  if (n <= 0) { return; }
  sort_keys_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, s>>>(e, n, id0, keys_in, ids_in, is_float ? 1 : 0);
  cub::DeviceRadixSort::SortPairs(temp, temp_bytes, keys_in, keys_out, ids_in, ids_out, n, 0, 32, s);
  const int64_t threads = n * static_cast<int64_t>(pitch / 16);
  place_sorted_kernel<<<static_cast<unsigned>((threads + 255) / 256), 256, 0, s>>>(
    keys_out, ids_out, n, row0, static_cast<const uint8_t*>(src), src_id0, pitch, static_cast<uint8_t*>(codes), perm, inv, init,
    metric, is_float ? 1 : 0);
}

void launch_kth_largest(const int32_t* gmax, int64_t ld, int ng, int k, int nq, int32_t* thr, cudaStream_t s,
                        const int32_t* ng_rows, int32_t never, int32_t* topk, const float* shift, uint32_t* zero)
{
  if (nq <= 0) { return; }
  if (topk == nullptr && ng <= kBitsHeld * 32 && k > 32) {
    kth_bits_kernel<<<(nq + 3) / 4, 128, 0, s>>>(gmax, ld, nq, ng, k, thr, ng_rows, never, shift, zero);
    return;
  }
  const size_t bytes = static_cast<size_t>(ng) * 4;
  constexpr size_t kMost = 160 * 1024;
  const int in_smem  = bytes <= kMost;
  if (in_smem) { allow_smem(kth_largest_kernel, bytes, kMost); }
  // short rows: smaller blocks, more of them per SM (the kernel is a chain of block-wide barriers)
  const int threads = ng > 4096 ? 512 : 2 * k <= 128 ? 128 : 2 * k <= 256 ? 256 : 512;
  kth_largest_kernel<<<nq, threads, in_smem ? bytes : 0, s>>>(gmax, ld, ng, k, thr, in_smem, ng_rows, never, topk, shift, zero);
}

void launch_remove(const int64_t* ids, int64_t n_ids, int64_t size, uint8_t* removed, int32_t* init, const int32_t* inv,
                   int32_t* cmax, bool is_float, unsigned long long* n_new, cudaStream_t s)
{
  if (n_ids <= 0) { return; }
  const auto grid     = static_cast<unsigned>((n_ids + 255) / 256);
  const int32_t never = is_float ? static_cast<int32_t>(0xff800000u) : kNeverInit;  // -inf or -2^30
  remove_kernel<<<grid, 256, 0, s>>>(ids, n_ids, size, removed, init, inv, n_new, never);
  if (init && cmax) { chain_max_of_ids_kernel<<<grid, 256, 0, s>>>(ids, n_ids, size, inv, init, cmax, is_float ? 1 : 0); }
}

int verify_launches(int dtype, int d, int k)
{
  const bool bytes = dtype == kI8 || dtype == kU8;
  return k > kSplitK || (!bytes && k > 32 && static_cast<size_t>(d) * dtype_size(dtype) >= kLongRow) ? 3 : 1;
}

void launch_verify_select(const void* vectors, size_t pitch, int dtype, int d, int metric, const void* queries,
                          size_t qpitch, int nq, int q0, const Candidates& cd, int k,
                          Admit adm, double* best_s, int32_t* best_row, int32_t* ovf_list, unsigned int* ovf_count,
                          unsigned long long* stats, Refine rf, cudaStream_t s, int32_t* kept, const int32_t* where, const double* sqnorm)
{
  if (nq <= 0) { return; }
  const int n2max  = cd.ld;
  const bool bytes = dtype == kI8 || dtype == kU8;  // 8-bit rows rank 64-bit keys
  const bool split = verify_launches(dtype, d, k) > 1;
  const size_t q_bytes = bytes ? static_cast<size_t>((d + 15) / 16 * 16) : sizeof(double) * static_cast<size_t>(d);
  const size_t pairs   = (sizeof(double) + sizeof(int32_t)) * static_cast<size_t>(n2max);
  // float rows: one staging tile per warp, + 16 bytes of alignment
  auto tiles = [&](int threads) { return bytes ? size_t(0) : 16 + static_cast<size_t>(threads / 32) * 32 * kStageStride; };
  by_dtype(dtype, [&](auto tag) {
    using T = decltype(tag);
    auto go = [&](auto kernel, dim3 grid, int threads, size_t smem) {
      // 2048 coordinates of a float query, lists of 4096, tiles of 8 warps
      constexpr size_t kMost = 8 * 2048 + 12 * 4096 + 16 + 8 * 32 * kStageStride;
      allow_smem(kernel, smem, kMost);
      kernel<<<grid, threads, smem, s>>>(static_cast<const uint8_t*>(vectors), pitch, d, queries, qpitch, q0, cd, n2max, k, adm,
                                         best_s, best_row, ovf_list, ovf_count, stats, rf, where, sqnorm, kept);
    };
    auto all = [&](auto metric, auto stored) {
      constexpr int M  = decltype(metric)::value;
      constexpr bool S = decltype(stored)::value;
      if (!split) {
        // a warp of float rows scores 32 rows at a time, and about k to 2 k are left to score
        const int threads = !bytes && k > 32 ? 256 : 128;
        go(verify_select_kernel<T, M, S, kFused>, dim3(nq), threads, q_bytes + pairs + tiles(threads));
        return;
      }
      // blocks by the length of the lists: the candidates of a query are a few times k, the rows to score one to two k
      const bool longer = k > kSplitK;
      go(verify_select_kernel<T, M, S, kRank>, dim3(nq), longer ? 1024 : 128, pairs);
      // (a batch has at most 32 768 queries: the second grid dimension takes them)
      const int threads = longer ? 128 : 64;
      const int pieces  = longer ? (n2max + threads - 1) / threads : (2 * k + threads - 1) / threads;
      go(verify_select_kernel<T, M, S, kScore>, dim3(pieces, nq), threads, q_bytes + tiles(threads));
      auto sort = [&](auto nt, auto held) {
        constexpr int NT = decltype(nt)::value, H = decltype(held)::value;
        const size_t smem = pairs + (4 * NT + 8) * sizeof(int32_t);
        allow_smem(sort_lists_kernel<T, M, NT, H>, smem, 12 * NT * H + (4 * NT + 8) * sizeof(int32_t));
        sort_lists_kernel<T, M, NT, H><<<nq, NT, smem, s>>>(queries, qpitch, d, q0, cd, n2max, k, best_s, best_row, ovf_list, ovf_count,
                                                            rf, kept);
      };
      if (n2max > 2048) {
        sort(std::integral_constant<int, 1024>{}, std::integral_constant<int, 4>{});
      } else {
        sort(std::integral_constant<int, 256>{}, std::integral_constant<int, 8>{});
      }
    };
    using std::integral_constant;
    if (metric == kL2) {
      all(integral_constant<int, kL2>{}, std::false_type{});
    } else if (metric == kIP) {
      all(integral_constant<int, kIP>{}, std::false_type{});
    } else if (sqnorm != nullptr && !bytes) {
      all(integral_constant<int, kCos>{}, std::true_type{});
    } else {
      all(integral_constant<int, kCos>{}, std::false_type{});
    }
  });
}

void launch_row_sqnorms(const void* vectors, size_t pitch, int dtype, int d, int64_t n, double* out, cudaStream_t s)
{
  if (n <= 0) { return; }
  const auto grid = static_cast<unsigned>((n + 127) / 128);
  if (dtype == kF16) {
    row_sqnorm_kernel<__half><<<grid, 128, 0, s>>>(static_cast<const uint8_t*>(vectors), pitch, d, n, out);
  } else {
    row_sqnorm_kernel<float><<<grid, 128, 0, s>>>(static_cast<const uint8_t*>(vectors), pitch, d, n, out);
  }
}

void launch_gather_rows(const void* in, size_t in_pitch, const int32_t* sel, int64_t n, int64_t n_pad, void* out,
                        size_t out_pitch, size_t row_bytes, cudaStream_t s)
{
  if (n_pad <= 0) { return; }
  const auto a    = reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out) | in_pitch | out_pitch | row_bytes;
  gather_rows_kernel<<<static_cast<unsigned>(n_pad), 128, 0, s>>>(static_cast<const uint8_t*>(in), in_pitch, sel, n,
                                                                   static_cast<uint8_t*>(out), out_pitch, row_bytes,
                                                                   (a & 15) == 0 ? 1 : 0);
}

void launch_to_half(const void* src, int kind, int64_t n, void* dst, int* bad, cudaStream_t s)
{
  if (n <= 0) { return; }
  const int aligned = ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15) == 0 ? 1 : 0;
  const auto grid   = static_cast<unsigned>(std::min<int64_t>((n / 8 + 255) / 256 + 1, 148 * 8));
  auto* h           = static_cast<__half*>(dst);
  if (kind == 0) {
    to_half_kernel<<<grid, 256, 0, s>>>(static_cast<const float*>(src), n, h, aligned, bad);
  } else if (kind == 1) {
    to_half_kernel<<<grid, 256, 0, s>>>(static_cast<const __half*>(src), n, h, aligned, bad);
  } else {
    to_half_kernel<<<grid, 256, 0, s>>>(static_cast<const __nv_bfloat16*>(src), n, h, aligned, bad);
  }
}

void launch_pack_mask(const uint8_t* mask, int64_t n, uint32_t* words, cudaStream_t s)
{
  if (n <= 0) { return; }
  pack_mask_kernel<<<static_cast<unsigned>(((n + 31) / 32 + 255) / 256), 256, 0, s>>>(mask, n, words,
                                                                                     (reinterpret_cast<uintptr_t>(mask) & 15) == 0);
}

void launch_label_rows(const int32_t* part_ids, int64_t n, const int64_t* off, const int64_t* lrow0, int n_labels,
                       const int32_t* inv, const int32_t* init, int32_t* lperm, int32_t* linv, int32_t* lsrc, int32_t* linit,
                       cudaStream_t s)
{
  if (n <= 0) { return; }
  label_rows_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, s>>>(part_ids, n, off, lrow0, n_labels, inv, init, lperm,
                                                                            linv, lsrc, linit);
}

void launch_scatter_best(const double* s2, const int32_t* row2, const int32_t* sel, int n, int k, double* best_s,
                         int32_t* best_row, cudaStream_t s)
{
  if (n <= 0) { return; }
  scatter_best_kernel<<<n, 128, 0, s>>>(s2, row2, sel, k, best_s, best_row);
}

void launch_compose(int32_t* list, const unsigned int* n, int n_max, const int32_t* sel, cudaStream_t s)
{
  if (n_max <= 0) { return; }
  compose_kernel<<<(n_max + 255) / 256, 256, 0, s>>>(list, n, sel);
}

void launch_dense_scores(const void* vectors, size_t pitch, int dtype, int d, int metric, int64_t n, const void* queries,
                         size_t qpitch, const int32_t* qsel, int q0, int nqb, Admit adm, double* out, int64_t ld,
                         cudaStream_t s)
{
  if (nqb <= 0 || n <= 0) { return; }
  const size_t smem = sizeof(double) * static_cast<size_t>(d) * kDenseQ;
  const dim3 grid(static_cast<unsigned>((n + 255) / 256), static_cast<unsigned>((nqb + kDenseQ - 1) / kDenseQ));
  by_dtype(dtype, [&](auto tag) {
    using T = decltype(tag);
    auto go = [&](auto kernel) {
      allow_smem(kernel, smem, kDenseMost);
      kernel<<<grid, 256, smem, s>>>(static_cast<const uint8_t*>(vectors), pitch, d, n, queries, qpitch, qsel, q0, nqb, adm, out, ld);
    };
    if (metric == kL2) {
      go(dense_scores_kernel<T, kL2>);
    } else if (metric == kIP) {
      go(dense_scores_kernel<T, kIP>);
    } else {
      go(dense_scores_kernel<T, kCos>);
    }
  });
}

namespace {
/// Rows of up to 8192 scores take blocks of 256 threads (many of them per SM), longer ones blocks of 1024.
template <typename... Args>
void launch_select(dim3 grid, int64_t n, const double* scores, int64_t ld, int64_t n_all, int k, Args... rest)
{
  auto go = [&](auto nt, const int32_t* qsel, int q0, double* best_s, int32_t* best_row, int64_t chunk, double* part_s, int32_t* part_row,
                const int64_t* row_off, const int32_t* row_n, cudaStream_t s) {
    constexpr int NT  = decltype(nt)::value;
    const size_t smem = select_smem<NT>(k);
    allow_smem(select_topk_kernel<NT>, smem, select_smem<NT>(2048));
    select_topk_kernel<NT><<<grid, NT, smem, s>>>(scores, ld, n_all, k, qsel, q0, best_s, best_row, chunk, part_s, part_row, row_off, row_n);
  };
  if (n <= 8192) {
    go(std::integral_constant<int, 256>{}, rest...);
  } else {
    go(std::integral_constant<int, 1024>{}, rest...);
  }
}
}  // namespace

void load_select_topk()
{
  cudaFuncAttributes a;
  cudaFuncGetAttributes(&a, select_topk_kernel<256>);
  cudaFuncGetAttributes(&a, select_topk_kernel<1024>);
  cudaFuncGetAttributes(&a, merge_partials_kernel);
}

int select_topk_parts(int64_t n, int k)
{
  // long rows are cut into chunks that separate blocks select from; at most 8192 partial winners per query
  if (n <= (1 << 18)) { return 1; }
  const int64_t by_size = (n + (1 << 17) - 1) >> 17;
  return static_cast<int>(std::max<int64_t>(1, std::min<int64_t>({by_size, 64, 8192 / k})));
}

void launch_select_topk(const double* scores, int64_t ld, int64_t n, int k, const int32_t* qsel, int q0, int nqb,
                        double* best_s, int32_t* best_row, double* part_s, int32_t* part_row, cudaStream_t s)
{
  if (nqb <= 0) { return; }
  const int parts   = select_topk_parts(n, k);
  if (parts == 1) {
    launch_select(dim3(nqb), n, scores, ld, n, k, qsel, q0, best_s, best_row, n, nullptr, nullptr, nullptr, nullptr, s);
    return;
  }
  const int64_t chunk = (n + parts - 1) / parts;
  launch_select(dim3(nqb, parts), chunk, scores, ld, n, k, qsel, q0, best_s, best_row, chunk, part_s, part_row, nullptr, nullptr, s);
  const int n2       = next_pow2(parts * k);
  const size_t smem2 = (sizeof(double) + sizeof(int32_t)) * static_cast<size_t>(n2);
  allow_smem(merge_partials_kernel, smem2, (sizeof(double) + sizeof(int32_t)) * 8192);
  merge_partials_kernel<<<nqb, 256, smem2, s>>>(part_s, part_row, parts, k, n2, qsel, q0, best_s, best_row);
}

void launch_select_topk_ragged(const double* scores, const int64_t* row_off, const int32_t* row_n, int64_t n_max, int k,
                               const int32_t* qsel, int nqb, double* best_s, int32_t* best_row, double* part_s,
                               int32_t* part_row, cudaStream_t s)
{
  if (nqb <= 0) { return; }
  const int parts   = select_topk_parts(n_max, k);
  if (parts == 1) {
    launch_select(dim3(nqb), n_max, scores, 0, 0, k, qsel, 0, best_s, best_row, std::max<int64_t>(n_max, 1), nullptr, nullptr, row_off,
                  row_n, s);
    return;
  }
  const int64_t chunk = (n_max + parts - 1) / parts;
  launch_select(dim3(nqb, parts), chunk, scores, 0, 0, k, qsel, 0, best_s, best_row, chunk, part_s, part_row, row_off, row_n, s);
  const int n2       = next_pow2(parts * k);
  const size_t smem2 = (sizeof(double) + sizeof(int32_t)) * static_cast<size_t>(n2);
  allow_smem(merge_partials_kernel, smem2, (sizeof(double) + sizeof(int32_t)) * 8192);
  merge_partials_kernel<<<nqb, 256, smem2, s>>>(part_s, part_row, parts, k, n2, qsel, 0, best_s, best_row);
}

void launch_dense_scores_grouped(const void* vectors, size_t pitch, int dtype, int d, int metric, const void* queries,
                                 size_t qpitch, const int32_t* order, const LabelGroup* groups, int n_groups,
                                 int64_t n_blocks, const int32_t* part_ids, int64_t tail0, int64_t n_tail, Admit adm,
                                 double* out, cudaStream_t s)
{
  if (n_groups <= 0 || n_blocks <= 0) { return; }
  const size_t smem = sizeof(double) * static_cast<size_t>(d) * kDenseQ;
  by_dtype(dtype, [&](auto tag) {
    using T = decltype(tag);
    auto go = [&](auto kernel) {
      allow_smem(kernel, smem, kDenseMost);
      kernel<<<static_cast<unsigned>(n_blocks), 256, smem, s>>>(static_cast<const uint8_t*>(vectors), pitch, d, queries, qpitch,
                                                                 order, groups, n_groups, part_ids, tail0, n_tail, adm, out);
    };
    if (metric == kL2) {
      go(dense_scores_grouped_kernel<T, kL2>);
    } else if (metric == kIP) {
      go(dense_scores_grouped_kernel<T, kIP>);
    } else {
      go(dense_scores_grouped_kernel<T, kCos>);
    }
  });
}

int64_t grouped_blocks(int nq, int64_t n_cols)
{
  return static_cast<int64_t>((nq + kDenseQ - 1) / kDenseQ) * ((n_cols + 255) / 256);
}

void launch_group_columns_to_ids(int32_t* best_row, int k, const int32_t* order, const LabelGroup* groups, int n_groups,
                                 const int32_t* part_ids, int64_t tail0, cudaStream_t s)
{
  if (n_groups <= 0) { return; }
  group_columns_to_ids_kernel<<<n_groups, 256, 0, s>>>(best_row, k, order, groups, part_ids, tail0);
}

// ids of all rows sorted by label (stable: ascending ids inside a label), the distinct labels and their counts
__global__ void iota_kernel(int32_t* p, int64_t n)
{
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < n) { p[i] = static_cast<int32_t>(i); }
}

// Order of the label-ordered copy of the screen's rows: by label, and inside a label by norm (the per-row term e of the
// screen), so that e is almost constant over 16 adjacent rows there too. keys [n]: (label, -e) of the partition
// entries; the sorted ids go to `order`. labels_of_ids: the label of every id; e is init[inv[id]].
__global__ void label_norm_keys_kernel(const int32_t* part_ids, int64_t n, const int32_t* labels_of_ids, const int32_t* inv,
                                       const int32_t* init, int is_float, unsigned long long* keys)
{
  const int64_t p = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (p >= n) { return; }
  const int32_t id   = part_ids[p];
  const int32_t e    = init[inv[id]];
  const uint32_t low = is_float ? __float_as_uint(-__int_as_float(e)) : static_cast<uint32_t>(-e);  // e <= 0
  const uint32_t top = static_cast<uint32_t>(labels_of_ids[id]) ^ 0x80000000u;                       // signed order
  keys[p]            = (static_cast<unsigned long long>(top) << 32) | low;
}

size_t label_norm_order_temp_bytes(int64_t n)
{
  size_t bytes = 0;
  cub::DeviceRadixSort::SortPairs(nullptr, bytes, static_cast<const unsigned long long*>(nullptr),
                                  static_cast<unsigned long long*>(nullptr), static_cast<const int32_t*>(nullptr),
                                  static_cast<int32_t*>(nullptr), n);
  return bytes;
}

void launch_label_norm_order(const int32_t* part_ids, int64_t n, const int32_t* labels_of_ids, const int32_t* inv,
                             const int32_t* init, bool is_float, unsigned long long* keys_in, unsigned long long* keys_out,
                             int32_t* order, void* temp, size_t temp_bytes, cudaStream_t s)
{
  if (n <= 0) { return; }
  label_norm_keys_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, s>>>(part_ids, n, labels_of_ids, inv, init,
                                                                                is_float ? 1 : 0, keys_in);
  cub::DeviceRadixSort::SortPairs(temp, temp_bytes, keys_in, keys_out, part_ids, order, n, 0, 64, s);
}

size_t label_partition_temp_bytes(int64_t n)
{
  size_t a = 0, b = 0;
  cub::DeviceRadixSort::SortPairs(nullptr, a, static_cast<const int32_t*>(nullptr), static_cast<int32_t*>(nullptr),
                                  static_cast<const int32_t*>(nullptr), static_cast<int32_t*>(nullptr), n);
  cub::DeviceRunLengthEncode::Encode(nullptr, b, static_cast<const int32_t*>(nullptr), static_cast<int32_t*>(nullptr),
                                     static_cast<int32_t*>(nullptr), static_cast<int32_t*>(nullptr), n);
  return std::max(a, b);
}

void launch_label_partition(const int32_t* labels, int64_t n, int32_t* labels_sorted, int32_t* ids_in, int32_t* part_ids,
                            int32_t* distinct, int32_t* counts, int32_t* n_distinct, void* temp, size_t temp_bytes,
                            cudaStream_t s)
{
  if (n <= 0) { return; }
  iota_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, s>>>(ids_in, n);
  cub::DeviceRadixSort::SortPairs(temp, temp_bytes, labels, labels_sorted, ids_in, part_ids, n, 0, 32, s);
  cub::DeviceRunLengthEncode::Encode(temp, temp_bytes, labels_sorted, distinct, counts, n_distinct, n, s);
}

namespace {
/// A thread per answer, as far as a block goes: with 64 threads the lists of 2048 took 32 turns, 23 us however few there were.
int finish_threads(int k) { return std::min(1024, std::max(64, (k + 31) / 32 * 32)); }
}  // namespace

void launch_finish(const double* best_s, const int32_t* best_row, int64_t id_base, const void* queries, size_t qpitch,
                   int dtype, int d, int metric, int nq, int k, int64_t* neighbors, float* distances, double* scores_out,
                   cudaStream_t s)
{
  if (nq <= 0) { return; }
  by_dtype(dtype, [&](auto tag) {
    using T = decltype(tag);
    finish_kernel<T><<<nq, finish_threads(k), 0, s>>>(best_s, best_row, nullptr, id_base, queries, qpitch, d, metric, k, neighbors, distances, scores_out);
  });
}

void launch_search_status(const unsigned int* count, const unsigned int* q_ovf, unsigned long long* status, cudaStream_t s)
{
  search_status_kernel<<<1, 1, 0, s>>>(count, q_ovf, status);
}

void launch_merge(const double* in_s, const int64_t* in_id, int parts, int nq, int k, const void* queries, size_t qpitch,
                  int dtype, int d, int metric, int64_t* neighbors, float* distances, double* scores_out, cudaStream_t s,
                  int64_t part_stride, bool finish)
{
  if (nq <= 0) { return; }
  if (part_stride == 0) { part_stride = static_cast<int64_t>(nq) * k; }
  // merged (score, id) go to scores_out / neighbors first; finish_kernel then converts in place
  if (parts * k <= kMergeSmallMax) {
    const int warps = 4;
    merge_small_kernel<<<(nq + warps - 1) / warps, warps * 32, static_cast<size_t>(warps) * parts * k * 16, s>>>(
      in_s, in_id, parts, nq, k, scores_out, neighbors, part_stride);
  } else {
    const int n2      = next_pow2(parts * k) < 2 ? 2 : next_pow2(parts * k);
    const size_t smem = (sizeof(double) + sizeof(int64_t)) * static_cast<size_t>(n2);
    allow_smem(merge_kernel, smem, (sizeof(double) + sizeof(int64_t)) * 8192);
    merge_kernel<<<nq, 256, smem, s>>>(in_s, in_id, parts, nq, k, n2, scores_out, neighbors, part_stride);
  }
  if (!finish) { return; }
  by_dtype(dtype, [&](auto tag) {
    using T = decltype(tag);
    finish_kernel<T><<<nq, finish_threads(k), 0, s>>>(scores_out, nullptr, neighbors, 0, queries, qpitch, d, metric, k, neighbors, distances, scores_out);
  });
}

}  // namespace certex_b200
