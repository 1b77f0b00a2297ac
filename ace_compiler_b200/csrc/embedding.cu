// The canonical embedding of the encoder and the decoder on the device.
//
// Same arithmetic as the host routines of the CPU runtime (util/src/ntt.c:598-675,
// ckks/src/encoder.c:268-292, 657-704), one IEEE operation at a time: complex
// products as four rounded multiplications and two rounded additions, no fused
// multiply-add anywhere (explicit _rn intrinsics), the roots of unity computed
// by the host's libm and uploaded in the order the stages read them.  The
// results are therefore the same doubles and the same rounded integers as the
// host routines produce.
//
// Both directions take two launches above 256 slots: the eight stages with
// spans below 256 on contiguous chunks of 256 points (one CTA each), the others
// on the columns of the (slots / 256) x 256 view, both in shared memory.  These
// kernels are latency bound (512 KiB of points at 32768 slots), so what counts
// is the number of launches and CTAs: one launch per wide stage and a last one
// of 8 CTAs with 4096 points each took 40 us, the two launches take 12.
//
// Decoding first puts every coefficient together from its residues (exact
// multiword arithmetic, one thread per coefficient) and truncates it to the 53
// bits the CPU runtime's big-integer conversion keeps.
#include <cmath>
#include <complex>
#include <cstring>
#include <map>
#include <vector>

#include "runtime.h"

namespace fhert {

namespace {

constexpr int64_t kMax64      = (int64_t)(((u64)1 << 63) - ((u64)1 << 9)) - 1;
constexpr int     kChunkLog   = 8;  // stages on contiguous chunks
constexpr int     kChunk      = 1 << kChunkLog;
constexpr int     kColumns    = 4;  // columns per CTA of the other stages

// constants of the reconstruction of a coefficient from `level` residues
struct CrtTable {
  int      words   = 0;        // of Q, one more for sums and the sign
  Twiddle* hat_inv = nullptr;  // [level] (Q / q_i)^-1 mod q_i
  u64*     hat     = nullptr;  // [level][words] Q / q_i
  u64*     q       = nullptr;  // [words] Q, then [words] floor(Q / 2)
  double*  recip   = nullptr;  // [level] 1 / q_i
};

struct EmbedTables {
  // stage with 2^(logm-1) butterflies per group: entries [2^(logm-1), 2^logm)
  double2* inv = nullptr;
  double2* fwd = nullptr;
  std::map<int, CrtTable>      crt;    // per level
  std::map<uint32_t, Twiddle*> scale;  // Delta^(d-1) modulo every prime, per degree d
};

__device__ __forceinline__ double2 add2(double2 a, double2 b) {
  return make_double2(__dadd_rn(a.x, b.x), __dadd_rn(a.y, b.y));
}
__device__ __forceinline__ double2 sub2(double2 a, double2 b) {
  return make_double2(__dsub_rn(a.x, b.x), __dsub_rn(a.y, b.y));
}
__device__ __forceinline__ double2 mul2(double2 a, double2 b) {
  return make_double2(__dsub_rn(__dmul_rn(a.x, b.x), __dmul_rn(a.y, b.y)),
                      __dadd_rn(__dmul_rn(a.x, b.y), __dmul_rn(a.y, b.x)));
}
// Gentleman-Sande (encoder) and Cooley-Tukey (decoder) butterflies
__device__ __forceinline__ void bfly_inv(double2& e, double2& o, double2 w) {
  const double2 d = sub2(e, o);
  e = add2(e, o);
  o = mul2(d, w);
}
__device__ __forceinline__ void bfly_fwd(double2& e, double2& o, double2 w) {
  const double2 t = mul2(w, o), x = e;
  e = add2(x, t);
  o = sub2(x, t);
}

enum InputKind { kComplex, kReal, kFloat };
template <int KIND>
__device__ __forceinline__ double2 input_point(const void* in, uint32_t p, uint32_t count) {
  if (p >= count) return make_double2(0.0, 0.0);
  if (KIND == kComplex) return static_cast<const double2*>(in)[p];
  if (KIND == kReal) return make_double2(static_cast<const double*>(in)[p], 0.0);
  return make_double2((double)static_cast<const float*>(in)[p], 0.0);
}

// ---- encoder -----------------------------------------------------------------

// stages with spans of 256 and more, on kColumns columns of 2^log_rows points
template <int KIND>
__global__ void __launch_bounds__(256)
embed_inv_columns(double2* __restrict__ v, const void* __restrict__ in, uint32_t count,
                  const double2* __restrict__ tw, int log_rows) {
  extern __shared__ double2 sh[];
  const int rows = 1 << log_rows, total = rows * kColumns;
  const uint32_t col = blockIdx.x * kColumns;
  for (int t = threadIdx.x; t < total; t += blockDim.x)
    sh[t] = input_point<KIND>(in, (uint32_t)(t / kColumns) * kChunk + col + t % kColumns, count);
  for (int l = log_rows; l > 0; l--) {
    __syncthreads();
    for (int t = threadIdx.x; t < total / 2; t += blockDim.x) {
      const int c = t % kColumns, b = t / kColumns, half = 1 << (l - 1);
      const int i = b & (half - 1), e = ((b >> (l - 1)) << l) + i;
      const uint32_t num2 = (uint32_t)half * kChunk;
      bfly_inv(sh[e * kColumns + c], sh[(e + half) * kColumns + c],
               __ldg(tw + num2 + (uint32_t)i * kChunk + col + c));
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < total; t += blockDim.x)
    v[(uint32_t)(t / kColumns) * kChunk + col + t % kColumns] = sh[t];
}

// The stages left, then the encoder's last step: bit reversal (point p goes to
// output index bit_reverse(p)), division by the length, scaling by Delta,
// rounding, and the split into the halves of the message polynomial.
template <int KIND>
__global__ void __launch_bounds__(kChunk / 2)
embed_inv_chunks(int64_t* __restrict__ msg, const void* __restrict__ in, uint32_t count,
                 const double2* __restrict__ tw, uint32_t slots, int log_slots, uint32_t gap,
                 double delta) {
  __shared__ double2 sh[kChunk];
  const int      k      = min(log_slots, kChunkLog);
  const uint32_t points = 1u << k, base = blockIdx.x * points;
  for (uint32_t p = threadIdx.x; p < points; p += blockDim.x)
    sh[p] = input_point<KIND>(in, base + p, count);
  for (int logm = k; logm > 0; logm--) {
    __syncthreads();
    const uint32_t num2 = 1u << (logm - 1);
    if (threadIdx.x < points / 2) {
      const uint32_t i = threadIdx.x & (num2 - 1), e = ((threadIdx.x >> (logm - 1)) << logm) + i;
      bfly_inv(sh[e], sh[e + num2], __ldg(tw + num2 + i));
    }
  }
  __syncthreads();
  const double d = (double)slots;
  for (uint32_t p = threadIdx.x; p < points; p += blockDim.x) {
    const uint32_t i  = log_slots ? (__brev(base + p) >> (32 - log_slots)) : 0;
    const double2  x  = sh[p];
    const double   re = __dadd_rn(__dmul_rn(__ddiv_rn(x.x, d), delta), 0.5);
    const double   im = __dadd_rn(__dmul_rn(__ddiv_rn(x.y, d), delta), 0.5);
    const int64_t  r = llround(re), m = llround(im);
    msg[(size_t)i * gap]           = r < 0 ? kMax64 + r : r;
    msg[(size_t)(i + slots) * gap] = m < 0 ? kMax64 + m : m;
  }
}

// ---- decoder -----------------------------------------------------------------

// Coefficient i of the polynomial as an integer in (-Q/2, Q/2], truncated to a
// double (encoder.c:657-690) and divided by the scaling factor.  W words: Q and
// one more.  With y_i = x_i (Q/q_i)^-1 mod q_i the integer is
// sum_i y_i Q/q_i - k Q, k = rint(sum_i y_i / q_i) unless that sum is close to a
// half, where exact comparisons decide.
template <int W>
__global__ void __launch_bounds__(128)
reconstruct_kernel(double* __restrict__ out, const u64* __restrict__ poly, CrtTable tab, int level,
                   const DevModulus* __restrict__ mods, uint32_t n, uint32_t slots, uint32_t gap,
                   double factor) {
  const uint32_t t = blockIdx.x * 128 + threadIdx.x;
  if (t >= 2 * slots) return;
  const uint32_t at = t < slots ? t * gap : n / 2 + (t - slots) * gap;
  typedef unsigned __int128 u128;
  u64    acc[W];
  double share = 0;
#pragma unroll
  for (int w = 0; w < W; w++) acc[w] = 0;
  const int words = tab.words;  // W is the next size there is a kernel for
  for (int i = 0; i < level; i++) {
    const Twiddle c = tab.hat_inv[i];
    const u64     y = mul_shoup(poly[(size_t)i * n + at], c.w, c.wp, mods[i].q);
    share += (double)y * tab.recip[i];
    u64 carry = 0;
#pragma unroll
    for (int w = 0; w < W; w++) {
      const u64  h = w < words ? __ldg(tab.hat + (size_t)i * words + w) : 0;
      const u128 p = (u128)y * h + acc[w] + carry;
      acc[w]       = (u64)p;
      carry        = (u64)(p >> 64);
    }
  }
  const double k    = rint(share);
  const u64    kq   = (u64)k;
  auto q_word = [&](int w) { return w < words ? __ldg(tab.q + w) : 0; };
  auto h_word = [&](int w) { return w < words ? __ldg(tab.q + words + w) : 0; };
  auto add_q  = [&](bool subtract, u64 times) {
    u64 carry = 0, borrow = 0;
#pragma unroll
    for (int w = 0; w < W; w++) {
      const u128 p = (u128)times * q_word(w) + carry;
      carry        = (u64)(p >> 64);
      const u64 v  = (u64)p;
      if (subtract) {
        const u64 r = acc[w] - v, b = acc[w] < v, s = r - borrow;
        borrow = b | (r < borrow);
        acc[w] = s;
      } else {
        const u64 r = acc[w] + v, b = r < v, s = r + borrow;
        borrow = b | (s < borrow);
        acc[w] = s;
      }
    }
  };
  auto over_half = [&]() {  // acc > floor(Q / 2), acc not negative
    int cmp = 0;
#pragma unroll
    for (int w = 0; w < W; w++) {
      const u64 h = h_word(w);
      if (acc[w] != h) cmp = acc[w] > h ? 1 : -1;
    }
    return cmp > 0;
  };
  add_q(true, kq);
  bool negative = (long long)acc[W - 1] < 0;
  if (fabs(share - k) > 0.499) {
    if (negative) add_q(false, 1);  // acc = the representative in [0, Q)
    negative = over_half();
    if (negative) add_q(true, 1);
  }
  if (negative) {
    u64 carry = 1;
#pragma unroll
    for (int w = 0; w < W; w++) {
      acc[w] = ~acc[w] + carry;
      carry  = carry && acc[w] == 0;
    }
  }
  // the top 53 bits of the magnitude
  int top = -1;
  u64 hi = 0, lo = 0;
#pragma unroll
  for (int w = 0; w < W; w++)
    if (acc[w] != 0) {
      top = w;
      hi  = acc[w];
      lo  = w > 0 ? acc[w - 1] : 0;
    }
  double v = 0.0;
  if (top >= 0) {
    const int lead  = __clzll(hi);
    const u64 bits  = lead ? (hi << lead) | (lo >> (64 - lead)) : hi;
    const int shift = top * 64 - lead;  // of the 64 leading bits
    v = top == 0 && lead >= 11 ? (double)hi : ldexp((double)(bits >> 11), shift + 11);
  }
  if (negative) v = -v;
  out[(t < slots ? 2 * t : 2 * (t - slots) + 1)] = __ddiv_rn(v, factor);
}

// stages with spans below 256, from the bit-reversed order
__global__ void __launch_bounds__(kChunk / 2)
embed_fwd_chunks(double2* __restrict__ out, const double2* __restrict__ v,
                 const double2* __restrict__ tw, int log_slots) {
  __shared__ double2 sh[kChunk];
  const int      k      = min(log_slots, kChunkLog);
  const uint32_t points = 1u << k, base = blockIdx.x * points;
  for (uint32_t p = threadIdx.x; p < points; p += blockDim.x)
    sh[p] = v[log_slots ? __brev(base + p) >> (32 - log_slots) : 0];
  for (int logm = 1; logm <= k; logm++) {
    __syncthreads();
    const uint32_t num = 1u << (logm - 1);
    if (threadIdx.x < points / 2) {
      const uint32_t i = threadIdx.x & (num - 1), e = ((threadIdx.x >> (logm - 1)) << logm) + i;
      bfly_fwd(sh[e], sh[e + num], __ldg(tw + num + i));
    }
  }
  __syncthreads();
  for (uint32_t p = threadIdx.x; p < points; p += blockDim.x) out[base + p] = sh[p];
}

// the others, on columns; `out` may be mapped host memory
__global__ void __launch_bounds__(256)
embed_fwd_columns(double2* __restrict__ out, const double2* __restrict__ v,
                  const double2* __restrict__ tw, int log_rows) {
  extern __shared__ double2 sh[];
  const int      rows = 1 << log_rows, total = rows * kColumns;
  const uint32_t col = blockIdx.x * kColumns;
  for (int t = threadIdx.x; t < total; t += blockDim.x)
    sh[t] = v[(uint32_t)(t / kColumns) * kChunk + col + t % kColumns];
  for (int l = 1; l <= log_rows; l++) {
    __syncthreads();
    for (int t = threadIdx.x; t < total / 2; t += blockDim.x) {
      const int c = t % kColumns, b = t / kColumns, half = 1 << (l - 1);
      const int i = b & (half - 1), e = ((b >> (l - 1)) << l) + i;
      bfly_fwd(sh[e * kColumns + c], sh[(e + half) * kColumns + c],
               __ldg(tw + (uint32_t)half * kChunk + (uint32_t)i * kChunk + col + c));
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < total; t += blockDim.x)
    out[(uint32_t)(t / kColumns) * kChunk + col + t % kColumns] = sh[t];
}

template <typename T>
T* to_device(const std::vector<T>& v) {
  T* d = nullptr;
  if (image_capturing()) image_capture_break("a table built on first use");
  CUDA_CHECK(cudaMalloc(&d, v.size() * sizeof(T)));
  CUDA_CHECK(cudaMemcpy(d, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice));
  CUDA_CHECK(cudaStreamSynchronize(0));  // fully on the device before the library stream reads it
  return d;
}

EmbedTables* tables_of(Context* c) {
  if (c->embed_tables != nullptr) return static_cast<EmbedTables*>(c->embed_tables);
  const size_t         m = 2ull * c->N, slots = c->N / 2;
  std::vector<double2> roots(m), inv(slots), fwd(slots);
  for (size_t i = 0; i < m; i++) {
    double angle = 2 * M_PI * i / m;
    roots[i]     = make_double2(std::cos(angle), std::sin(angle));
  }
  std::vector<uint32_t> rot(slots);
  rot[0] = 1;
  for (size_t i = 1; i < slots; i++) rot[i] = (uint32_t)((5ull * rot[i - 1]) % m);
  for (size_t num = 1; num < slots; num <<= 1) {  // ntt.c:612-621, 646-655
    const size_t order = num << 3, gap = m / order;
    for (size_t i = 0; i < num; i++) {
      fwd[num + i] = roots[(rot[i] % order) * gap];
      inv[num + i] = roots[(order - rot[i] % order) * gap];
    }
  }
  EmbedTables* t  = new EmbedTables();
  t->inv          = to_device(inv);
  t->fwd          = to_device(fwd);
  c->embed_tables = t;
  return t;
}

// little-endian multiword: acc += a * m
void big_mul_add(std::vector<u64>& acc, const std::vector<u64>& a, u64 m) {
  u64 carry = 0;
  for (size_t i = 0; i < acc.size(); i++) {
    u128 t = (u128)(i < a.size() ? a[i] : 0) * m + acc[i] + carry;
    acc[i] = (u64)t;
    carry  = (u64)(t >> 64);
  }
}

const CrtTable& crt_table(Context* c, int level) {
  auto& all = tables_of(c)->crt;
  auto  it  = all.find(level);
  if (it != all.end()) return it->second;
  // product of the first `level` primes without prime `skip`
  auto product = [&](int skip) {
    std::vector<u64> p(level + 1, 0);
    p[0] = 1;
    for (int k = 0; k < level; k++) {
      if (k == skip) continue;
      std::vector<u64> next(level + 1, 0);
      big_mul_add(next, p, c->primes[k]);
      p.swap(next);
    }
    return p;
  };
  std::vector<u64> q = product(-1);
  int              words = level + 1;
  while (words > 1 && q[words - 1] == 0) words--;
  std::vector<Twiddle> hat_inv(level);
  std::vector<u64>     hat((size_t)level * words), qs(2 * (size_t)words);
  std::vector<double>  recip(level);
  for (int i = 0; i < level; i++) {
    const u64        qi = c->primes[i];
    std::vector<u64> p  = product(i);
    std::copy(p.begin(), p.begin() + words, hat.begin() + (size_t)i * words);
    u64 h = 1;
    for (int k = 0; k < level; k++)
      if (k != i) h = mulmod(h, c->primes[k] % qi, qi);
    hat_inv[i].w  = invmod(h, qi);
    hat_inv[i].wp = shoup(hat_inv[i].w, qi);
    recip[i]      = 1.0 / (double)qi;
  }
  for (int w = 0; w < words; w++) {
    qs[w]         = q[w];
    qs[words + w] = (q[w] >> 1) | (w + 1 < words ? q[w + 1] << 63 : 0);
  }
  CrtTable t;
  t.words   = words;
  t.hat_inv = to_device(hat_inv);
  t.hat     = to_device(hat);
  t.q       = to_device(qs);
  t.recip   = to_device(recip);
  return all.emplace(level, t).first->second;
}

size_t column_smem(int log_rows) { return ((size_t)kColumns << log_rows) * sizeof(double2); }

template <typename K>
void allow_smem(K kernel, size_t bytes) {
  if (bytes > 48 * 1024)
    CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
}

template <int KIND>
void embed_inverse(Context* c, const EmbedTables* t, const void* in, size_t count, uint32_t slots,
                   int64_t* msg) {
  const uint32_t n = c->N, gap = n / (slots * 2);
  int            lg = 0;
  while ((1u << lg) < slots) lg++;
  const double delta = std::pow(2.0, (double)c->sf_bits);
  prof_before(KID_ENCODE);
  if (lg <= kChunkLog) {
    launch(embed_inv_chunks<KIND>, 1, kChunk / 2, 0, c->stream, msg, in, (uint32_t)count, t->inv,
           slots, lg, gap, delta);
  } else {
    double2* v = nullptr;
    CUDA_CHECK(dev_alloc(&v, (size_t)slots * sizeof(double2), c->stream));
    const size_t smem = column_smem(lg - kChunkLog);
    allow_smem(embed_inv_columns<KIND>, smem);
    launch(embed_inv_columns<KIND>, kChunk / kColumns, 256, smem, c->stream, v, in, (uint32_t)count,
           t->inv, lg - kChunkLog);
    launch(embed_inv_chunks<kComplex>, slots >> kChunkLog, kChunk / 2, 0, c->stream, msg,
           (const void*)v, slots, t->inv, slots, lg, gap, delta);
    c->launches++;
    CUDA_CHECK(dev_free(v, c->stream));
  }
  c->launches++;
  prof_after(KID_ENCODE, 1);
  CUDA_CHECK(cudaGetLastError());
}

template <int W>
bool reconstruct(Context* c, const CrtTable& tab, double* out, const u64* poly, int level,
                 uint32_t slots, uint32_t gap, double factor) {
  if (tab.words + 1 > W) return false;
  launch(reconstruct_kernel<W>, (2 * slots + 127) / 128, 128, 0, c->stream, out, poly, tab, level,
         c->d_mod, c->N, slots, gap, factor);
  c->launches++;
  return true;
}

}  // namespace

void free_embed_tables(Context* c) {
  if (c->embed_tables == nullptr) return;
  EmbedTables* t = static_cast<EmbedTables*>(c->embed_tables);
  cudaFree(t->inv);
  cudaFree(t->fwd);
  for (auto& kv : t->crt) {
    cudaFree(kv.second.hat_inv);
    cudaFree(kv.second.hat);
    cudaFree(kv.second.q);
    cudaFree(kv.second.recip);
  }
  for (auto& kv : t->scale) cudaFree(kv.second);
  delete t;
  c->embed_tables = nullptr;
}

const Twiddle* scale_powers(Context* c, uint32_t degree) {
  auto& all = tables_of(c)->scale;
  auto  it  = all.find(degree);
  if (it != all.end()) return it->second;
  // Delta^(d-1) modulo every Q prime (encoder.c:297-312); the special limbs keep
  // the message as it is
  std::vector<Twiddle> pow(c->primes.size());
  const u64            delta = (u64)(int64_t)std::pow(2.0, (double)c->sf_bits);
  for (size_t i = 0; i < pow.size(); i++) {
    const u64 q = c->primes[i];
    u64       p = 1 % q;
    if ((int)i < c->L)
      for (uint32_t d = 1; d < degree; d++) p = mulmod(p, delta % q, q);
    pow[i].w  = p;
    pow[i].wp = shoup(p, q);
  }
  return all[degree] = to_device(pow);
}

void encode_message_on_device(Context* c, const MessageInput& in, uint32_t slots, int64_t* d_msg) {
  EmbedTables* t    = tables_of(c);
  const size_t size = in.kind == MessageInput::kFloats ? sizeof(float)
                      : in.kind == MessageInput::kReals ? sizeof(double)
                                                        : sizeof(double2);
  void* d_in = nullptr;
  CUDA_CHECK(dev_alloc(&d_in, std::max<size_t>(1, in.count * size), c->stream));
  upload_staged(c, d_in, in.data, in.count * size);
  if (c->N / (slots * 2) > 1)  // zeros between the used coefficients
    CUDA_CHECK(zero_async(d_msg, (size_t)c->N * sizeof(int64_t), c->stream));
  if (in.kind == MessageInput::kFloats) embed_inverse<kFloat>(c, t, d_in, in.count, slots, d_msg);
  else if (in.kind == MessageInput::kReals) embed_inverse<kReal>(c, t, d_in, in.count, slots, d_msg);
  else embed_inverse<kComplex>(c, t, d_in, in.count, slots, d_msg);
  CUDA_CHECK(dev_free(d_in, c->stream));
}

void decode_on_device(Context* c, const int64_t* poly, int level, uint32_t slots, double factor,
                      double* out, size_t count) {
  EmbedTables*    t   = tables_of(c);
  const CrtTable& tab = crt_table(c, level);
  const uint32_t  gap = c->N / 2 / slots;
  int             lg  = 0;
  while ((1u << lg) < slots) lg++;
  double2 *v = nullptr, *u = nullptr;
  const size_t bytes = (size_t)slots * sizeof(double2);
  CUDA_CHECK(dev_alloc(&v, bytes, c->stream));
  CUDA_CHECK(dev_alloc(&u, bytes, c->stream));
  const u64* src = reinterpret_cast<const u64*>(poly);
  double*    dv  = reinterpret_cast<double*>(v);
  prof_before(KID_ENCODE);
  const bool done = reconstruct<3>(c, tab, dv, src, level, slots, gap, factor) ||
                    reconstruct<6>(c, tab, dv, src, level, slots, gap, factor) ||
                    reconstruct<10>(c, tab, dv, src, level, slots, gap, factor) ||
                    reconstruct<18>(c, tab, dv, src, level, slots, gap, factor) ||
                    reconstruct<36>(c, tab, dv, src, level, slots, gap, factor) ||
                    reconstruct<98>(c, tab, dv, src, level, slots, gap, factor);
  FHERT_ASSERT(done, "decoding from %d limbs unsupported", level);
  // the last launch writes into pinned host memory
  double2* host = static_cast<double2*>(pinned_output(c, bytes));
  if (lg <= kChunkLog) {
    launch(embed_fwd_chunks, 1, kChunk / 2, 0, c->stream, host, v, t->fwd, lg);
  } else {
    launch(embed_fwd_chunks, slots >> kChunkLog, kChunk / 2, 0, c->stream, u, v, t->fwd, lg);
    const size_t smem = column_smem(lg - kChunkLog);
    allow_smem(embed_fwd_columns, smem);
    launch(embed_fwd_columns, kChunk / kColumns, 256, smem, c->stream, host, u, t->fwd, lg - kChunkLog);
    c->launches++;
  }
  c->launches++;
  prof_after(KID_ENCODE, 1);
  CUDA_CHECK(cudaGetLastError());
  CUDA_CHECK(dev_free(v, c->stream));
  CUDA_CHECK(dev_free(u, c->stream));
  CUDA_CHECK(stream_sync(c->stream));
  c->d2h_bytes += bytes;
  std::memcpy(out, host, count * sizeof(double2));
}

// ---- host memory the device reads and writes -----------------------------------
//
// A copy from pageable memory makes the driver stage it and often wait for it.
// What an entry point takes from its caller goes through a ring of pinned
// buffers instead: one memory copy on the host, then a copy kernel among the
// gathered launches.  A buffer is used again once the work queued behind its
// last use is done.

namespace {
struct Pinned {
  void*       p     = nullptr;
  size_t      bytes = 0;
  cudaEvent_t used  = nullptr;
  bool        busy  = false;
};
struct HostBuffers {
  static constexpr int kRing = 8;
  Pinned   ring[kRing];
  unsigned next = 0;
  Pinned*  last = nullptr;  // its use has been queued, not yet marked
  Pinned   out;
};
HostBuffers* host_buffers(Context* c) {
  if (c->host_buffers == nullptr) c->host_buffers = new HostBuffers();
  return static_cast<HostBuffers*>(c->host_buffers);
}
void grow(Pinned& b, size_t bytes) {
  if (b.bytes >= bytes) return;
  if (b.p) cudaFreeHost(b.p);
  b.bytes = std::max<size_t>(bytes, 64 * 1024);
  CUDA_CHECK(cudaHostAlloc(&b.p, b.bytes, cudaHostAllocMapped | cudaHostAllocPortable));
}
}  // namespace

void upload_staged(Context* c, void* dst, const void* src, size_t bytes) {
  if (bytes == 0) return;
  if (image_capturing()) {  // a captured copy reads its own snapshot
    CUDA_CHECK(counted_copy(dst, src, bytes, cudaMemcpyHostToDevice, c->stream));
    return;
  }
  HostBuffers* h = host_buffers(c);
  if (h->last != nullptr) {
    launch_flush();
    CUDA_CHECK(cudaEventRecord(h->last->used, c->stream));
    h->last->busy = true;
    h->last       = nullptr;
  }
  Pinned& b = h->ring[h->next++ % HostBuffers::kRing];
  if (b.used == nullptr) CUDA_CHECK(cudaEventCreateWithFlags(&b.used, cudaEventDisableTiming));
  if (b.busy) {
    CUDA_CHECK(cudaEventSynchronize(b.used));
    b.busy = false;
  }
  const size_t padded = (bytes + 15) & ~(size_t)15;  // device blocks are multiples of 256 bytes
  grow(b, padded);
  std::memcpy(b.p, src, bytes);
  c->h2d_bytes += bytes;
  if (!launch_copy(dst, b.p, padded, c->stream))
    CUDA_CHECK(cudaMemcpyAsync(dst, b.p, bytes, cudaMemcpyHostToDevice, c->stream));
  h->last = &b;
}

void* pinned_output(Context* c, size_t bytes) {
  HostBuffers* h = host_buffers(c);
  grow(h->out, bytes);
  return h->out.p;
}

void free_host_buffers(Context* c) {
  if (c->host_buffers == nullptr) return;
  HostBuffers* h = static_cast<HostBuffers*>(c->host_buffers);
  for (Pinned& b : h->ring) {
    if (b.p) cudaFreeHost(b.p);
    if (b.used) cudaEventDestroy(b.used);
  }
  if (h->out.p) cudaFreeHost(h->out.p);
  delete h;
  c->host_buffers = nullptr;
}

}  // namespace fhert
