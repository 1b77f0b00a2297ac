// Sums of products over digits, rotations and plaintexts: the key inner product
// and the sums of the bootstrapping transforms (rns_poly.c:516,
// rns_poly_impl.c:13-160, ckks/src/bootstrap.c:1233-1373).
//
// All of them stream their operands from HBM, each word feeding one or two
// multiply-adds, so what matters is that every operand is read once, that
// enough bytes are in flight, and that what follows (a permutation, an addition)
// happens before the result is written.  Two coefficients per thread (16-byte
// loads), one reduction per output word.
#include <algorithm>
#include <array>
#include <type_traits>

#include "ntt_kernels.cuh"
#include "runtime.h"

namespace fhert {

namespace {

constexpr int kThreads = 256;
constexpr int kTile    = 256;  // coefficients per CTA where blocks are permuted: one block

// Sums of products of residues.  Few: at most four products; else at most 16.
//   SumFp     primes transformed in double precision: every product is reduced at
//             once (6 operations of the double-precision pipe), sums stay below
//             13p.  A key inner product of three digits takes 56 cycles of that
//             pipe per word; carry-free halves take 66 cycles of the integer
//             multiplier and 70 more for the reduction.
//   SumHalves all primes below 2^60: four accumulators of 30-bit halves, no
//             carries, one reduction
//   SumWide   128-bit words
struct SumFp {
  struct Mod {
    nttk::ArithFp ar;
    __device__ __forceinline__ explicit Mod(const DevModulus& m) : ar(m) {}
  };
  typedef double Word;  // an operand
  double         v;
  static __device__ __forceinline__ Word word(u64 x) { return nttk::ArithFp::load(x); }
  __device__ __forceinline__ void zero() { v = 0; }
  __device__ __forceinline__ void mac(Word x, Word y, const Mod& m) { v = __dadd_rn(v, m.ar.mul(x, y)); }
  template <bool FEW>
  __device__ __forceinline__ u64 value(const Mod& m, const DevModulus&) const { return m.ar.canon(v); }
};
struct SumHalves {
  struct Mod {
    __device__ __forceinline__ explicit Mod(const DevModulus&) {}
  };
  struct Word {
    uint32_t lo, hi;
  };
  Acc4 a;
  static __device__ __forceinline__ Word word(u64 x) {
    return Word{(uint32_t)x & 0x3fffffffu, (uint32_t)(x >> 30)};
  }
  __device__ __forceinline__ void zero() { acc4_zero(a); }
  __device__ __forceinline__ void mac(Word x, Word y, const Mod&) { acc4_mac_halves(a, x.lo, x.hi, y.lo, y.hi); }
  template <bool FEW>
  __device__ __forceinline__ u64 value(const Mod&, const DevModulus& m) const {
    u64 hi, lo;
    acc4_fold(a, hi, lo);
    return FEW ? reduce_few(hi, lo, m) : reduce_128(hi, lo, m);
  }
};
struct SumWide {
  struct Mod {
    __device__ __forceinline__ explicit Mod(const DevModulus&) {}
  };
  typedef u64 Word;
  u64         hi, lo;
  static __device__ __forceinline__ Word word(u64 x) { return x; }
  __device__ __forceinline__ void zero() { hi = lo = 0; }
  __device__ __forceinline__ void mac(Word x, Word y, const Mod&) { mac_128(hi, lo, x, y); }
  template <bool FEW>
  __device__ __forceinline__ u64 value(const Mod&, const DevModulus& m) const { return reduce_128(hi, lo, m); }
};

__device__ __forceinline__ ulonglong2 load2(const u64* p, uint32_t pair) {
  return reinterpret_cast<const ulonglong2*>(p)[pair];
}
// read once per key switch: past the lines that tables and polynomials in flight
// should keep
__device__ __forceinline__ ulonglong2 stream2(const u64* p, uint32_t pair) {
  return __ldcs(reinterpret_cast<const ulonglong2*>(p) + pair);
}

// *p = v, or *p += v mod q
__device__ __forceinline__ void put1(u64* p, u64 v, bool accumulate, u64 q) {
  *p = accumulate ? add_mod(*p, v, q) : v;
}
__device__ __forceinline__ void put2(u64* p, ulonglong2 v, bool accumulate, u64 q) {
  ulonglong2* w = reinterpret_cast<ulonglong2*>(p);
  if (accumulate) {
    const ulonglong2 o = *w;
    v = make_ulonglong2(add_mod(o.x, v.x, q), add_mod(o.y, v.y, q));
  }
  *w = v;
}

struct LimbList {  // limbs covered by a launch, blockIdx.y -> limb
  int     count;
  bool    is_float;
  uint8_t limb[kMaxLimbs / 2];
};

// ---- one pair of sums: acc = sum_j e_j * key_j ----------------------------------
//
// The digits are taken U at a time and all operands of a group are loaded
// before the first multiply; registers are capped for four CTAs per SM (84 us
// at 36 limbs with two CTAs, 44 with four: 6.0 TB/s).  EXACT: there are exactly
// U digits (the key switch: up to four); else any number, in groups of U (a
// group that reaches past the last digit loads nothing for the missing ones and
// multiplies zeros).
template <bool TWO, class S, int U, bool EXACT>
__global__ void __launch_bounds__(kThreads, 4)
inner_product_kernel(const __grid_constant__ InnerArgs a, const __grid_constant__ LimbList list, int num_q, const DevModulus* __restrict__ mods,
                     uint32_t n) {
  const int        m     = list.limb[blockIdx.y];  // among level Q limbs then K P limbs
  const bool       is_q  = m < a.level;
  const int        prime = is_q ? m : num_q + (m - a.level);
  const DevModulus md    = mods[prime];
  const size_t e_off = (size_t)(is_q ? m : a.ext_p_limb + (m - a.level)) * n;
  const size_t k_off = (size_t)(is_q ? m : a.key_p_limb + (m - a.level)) * n;
  const size_t d_off = (size_t)(is_q ? m : a.acc_p_limb + (m - a.level)) * n;
  const int    own   = (a.in != nullptr && is_q) ? m / a.alpha : -1;
  const typename S::Mod sm(md);
  const uint32_t pairs = n >> 1;
  for (uint32_t i = blockIdx.x * kThreads + threadIdx.x; i < pairs; i += gridDim.x * kThreads) {
    S s[4];
#pragma unroll
    for (int k = 0; k < 4; k++) s[k].zero();
#pragma unroll 1
    for (int base = 0; base < (EXACT ? U : a.parts); base += U) {
      ulonglong2 e[U], k0[U], k1[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int j = base + u;
        if (!EXACT) e[u] = k0[u] = k1[u] = make_ulonglong2(0, 0);
        if (EXACT || j < a.parts) {
          const u64* es = (j == own) ? a.in + (size_t)m * n : a.ext_ptr[j] + e_off;
          e[u]  = load2(es, i);
          k0[u] = stream2(a.key0[j] + k_off, i);
          if (TWO) k1[u] = stream2(a.key1[j] + k_off, i);
        }
      }
#pragma unroll
      for (int u = 0; u < U; u++) {
        const typename S::Word ex = S::word(e[u].x), ey = S::word(e[u].y);
        s[0].mac(ex, S::word(k0[u].x), sm);
        s[1].mac(ey, S::word(k0[u].y), sm);
        if (TWO) {
          s[2].mac(ex, S::word(k1[u].x), sm);
          s[3].mac(ey, S::word(k1[u].y), sm);
        }
      }
    }
    ulonglong2 v0 = make_ulonglong2(s[0].template value<EXACT>(sm, md), s[1].template value<EXACT>(sm, md));
    ulonglong2 v1{};
    if (TWO) v1 = make_ulonglong2(s[2].template value<EXACT>(sm, md), s[3].template value<EXACT>(sm, md));
    if (TWO && a.add[0] != nullptr && is_q) {
      const Twiddle    p  = a.p_mod_q[m];
      const ulonglong2 x0 = load2(a.add[0] + d_off, i), x1 = load2(a.add[1] + d_off, i);
      v0.x = add_mod(v0.x, mul_shoup(x0.x, p.w, p.wp, md.q), md.q);
      v0.y = add_mod(v0.y, mul_shoup(x0.y, p.w, p.wp, md.q), md.q);
      v1.x = add_mod(v1.x, mul_shoup(x1.x, p.w, p.wp, md.q), md.q);
      v1.y = add_mod(v1.y, mul_shoup(x1.y, p.w, p.wp, md.q), md.q);
    }
    reinterpret_cast<ulonglong2*>(a.acc0 + d_off)[i] = v0;
    if (TWO) reinterpret_cast<ulonglong2*>(a.acc1 + d_off)[i] = v1;
  }
}

// ---- the same digits against several keys ---------------------------------------
//
// Rotations of one ciphertext share their raised digits: they stay in registers
// while the keys of all rotations stream by, and each result is permuted (a
// polynomial, perhaps lifted by P, having been added to the first) on its way
// out, where it may join what is there already.  The permutation sends blocks of 256 to
// blocks of 256, so a CTA with a whole source block permutes in shared memory
// and writes a whole destination block.  At 44 limbs a rotation took an inner
// product (41 us) and a gather with addition (24 us); here it is its key's 264
// limbs read and 88 written, 30 us.
template <class S, int U, bool EXACT>
__global__ void __launch_bounds__(kTile / 2, EXACT ? 6 : 1)
keys_product_kernel(const __grid_constant__ KeysArgs a, const __grid_constant__ LimbList list, int num_q, const DevModulus* __restrict__ mods,
                    uint32_t n) {
  __shared__ __align__(16) u64 sh[2][2][kTile];
  const int        m     = list.limb[blockIdx.y];
  const bool       is_q  = m < a.level;
  const int        prime = is_q ? m : num_q + (m - a.level);
  const DevModulus md    = mods[prime];
  const size_t     off   = (size_t)m * n;  // of the digits and the results
  const size_t     k_off = (size_t)(is_q ? m : a.key_p_limb + (m - a.level)) * n;
  const int        own   = is_q ? m / a.alpha : -1;
  const uint32_t   i     = blockIdx.x * (kTile / 2) + threadIdx.x;  // pair of coefficients
  if (n < (uint32_t)kTile && i >= n / 2) return;
  const typename S::Mod sm(md);
  ulonglong2            e[U];
#pragma unroll
  for (int j = 0; j < U; j++)
    if (EXACT || j < a.parts) e[j] = load2(j == own ? a.in + off : a.digits + (size_t)j * a.digit_stride + off, i);
  ulonglong2 more = make_ulonglong2(0, 0);
  if (a.c0 != nullptr && (is_q || a.p_mod_q == nullptr)) {
    more = load2(a.c0 + off, i);
    if (a.p_mod_q != nullptr) {
      const Twiddle p = a.p_mod_q[m];
      more = make_ulonglong2(mul_shoup(more.x, p.w, p.wp, md.q), mul_shoup(more.y, p.w, p.wp, md.q));
    }
  }
#pragma unroll 1
  for (int r = 0; r < a.count; r++) {
    ulonglong2 k0[U], k1[U];
#pragma unroll
    for (int j = 0; j < U; j++) {
      if (!EXACT && j >= a.parts) break;
      k0[j] = stream2(a.key0[r][j] + k_off, i);
      k1[j] = stream2(a.key1[r][j] + k_off, i);
    }
    S s[4];
#pragma unroll
    for (int k = 0; k < 4; k++) s[k].zero();
#pragma unroll
    for (int j = 0; j < U; j++) {
      if (!EXACT && j >= a.parts) break;
      const typename S::Word ex = S::word(e[j].x), ey = S::word(e[j].y);
      s[0].mac(ex, S::word(k0[j].x), sm);
      s[1].mac(ey, S::word(k0[j].y), sm);
      s[2].mac(ex, S::word(k1[j].x), sm);
      s[3].mac(ey, S::word(k1[j].y), sm);
    }
    const ulonglong2 v0 = make_ulonglong2(add_mod(s[0].template value<EXACT>(sm, md), more.x, md.q),
                                          add_mod(s[1].template value<EXACT>(sm, md), more.y, md.q));
    const ulonglong2 v1  = make_ulonglong2(s[2].template value<EXACT>(sm, md), s[3].template value<EXACT>(sm, md));
    u64*             out = a.out + (size_t)r * a.out_stride;
    if (a.place[r] == nullptr) {
      put2(out + off + 2 * (size_t)i, v0, a.accumulate, md.q);
      put2(out + a.poly_stride + off + 2 * (size_t)i, v1, a.accumulate, md.q);
      continue;
    }
    // place[s] = destination of source coefficient s
    const uint2 to = reinterpret_cast<const uint2*>(a.place[r])[i];
    if (n < (uint32_t)kTile) {
      put1(out + off + to.x, v0.x, a.accumulate, md.q);
      put1(out + off + to.y, v0.y, a.accumulate, md.q);
      put1(out + a.poly_stride + off + to.x, v1.x, a.accumulate, md.q);
      put1(out + a.poly_stride + off + to.y, v1.y, a.accumulate, md.q);
      continue;
    }
    u64(&turn)[2][kTile] = sh[r & 1];  // what the turn before left is still being read
    turn[0][to.x & 255]  = v0.x;
    turn[0][to.y & 255]  = v0.y;
    turn[1][to.x & 255]  = v1.x;
    turn[1][to.y & 255]  = v1.y;
    __syncthreads();
    const size_t dst = off + (to.x & ~255u) + 2 * threadIdx.x;
    put2(out + dst, *reinterpret_cast<const ulonglong2*>(&turn[0][2 * threadIdx.x]), a.accumulate, md.q);
    put2(out + a.poly_stride + dst, *reinterpret_cast<const ulonglong2*>(&turn[1][2 * threadIdx.x]),
         a.accumulate, md.q);
  }
}

// eight sums of halves take 64 registers, of doubles 16
template <class S>
constexpr int kWeightedCtas = 2;
template <>
constexpr int kWeightedCtas<SumFp> = 2;

// ---- several plaintext-weighted sums of the same rotations ------------------------
//
// out_i = sum_j rot_j * plain_{i,j} for up to four baby steps i at once, both
// polynomials: every rotation is read once for all of them.  One coefficient per
// thread keeps the eight sums in registers.  (One baby step per launch read the
// rotations of 44 limbs four times: 146 us each, 7.5 TB/s.)
template <class S, int B>
__global__ void __launch_bounds__(kThreads, kWeightedCtas<S>)
weighted_sums_kernel(const __grid_constant__ SumsArgs a, const __grid_constant__ LimbList list, int num_q, const DevModulus* __restrict__ mods,
                     uint32_t n) {
  const int        m     = list.limb[blockIdx.y];
  const bool       is_q  = m < a.level;
  const DevModulus md    = mods[is_q ? m : num_q + (m - a.level)];
  const size_t     off   = (size_t)m * n + blockIdx.x * kThreads + threadIdx.x;
  if (blockIdx.x * kThreads + threadIdx.x >= n) return;
  const size_t     p_off = off - (size_t)m * n;  // coefficient
  const typename S::Mod sm(md);
  S                s[B][2];
#pragma unroll
  for (int i = 0; i < B; i++)
#pragma unroll
    for (int k = 0; k < 2; k++) s[i][k].zero();
  // operands of two terms are on their way while the two before are multiplied
  struct Operands {
    u64 r0, r1, w[B];
  };
  auto fetch = [&](Operands& o, int j) {
    const bool here = j < a.terms;
    const u64* r    = a.rot + (size_t)j * a.rot_stride + off;
    o.r0 = here ? r[0] : 0;
    o.r1 = here ? r[a.poly_stride] : 0;
#pragma unroll
    for (int i = 0; i < B; i++) {
      const SumsArgs::Plain p = a.plain[i][here ? j : 0];
      const size_t row = is_q ? (size_t)m : (size_t)(p.p_limb + m - a.level);
      o.w[i] = here && p.data != nullptr ? __ldcs(p.data + row * n + p_off) : 0;
    }
  };
  auto multiply = [&](const Operands& o) {
    const typename S::Word r0 = S::word(o.r0), r1 = S::word(o.r1);
#pragma unroll
    for (int i = 0; i < B; i++) {
      const typename S::Word w = S::word(o.w[i]);
      s[i][0].mac(r0, w, sm);
      s[i][1].mac(r1, w, sm);
    }
  };
  Operands x[2], y[2];
  fetch(x[0], 0);
  fetch(x[1], 1);
#pragma unroll 1
  for (int j = 0; j < a.terms; j += 4) {
    fetch(y[0], j + 2);
    fetch(y[1], j + 3);
    multiply(x[0]);
    multiply(x[1]);
    fetch(x[0], j + 4);
    fetch(x[1], j + 5);
    multiply(y[0]);
    multiply(y[1]);
  }
#pragma unroll
  for (int i = 0; i < B; i++) {
    u64* out = a.out + (size_t)i * a.out_stride + off;
    out[0]             = s[i][0].template value<false>(sm, md);
    out[a.poly_stride] = s[i][1].template value<false>(sm, md);
  }
}

// ---- sums of ciphertexts times constants ------------------------------------------
//
// out = sum_j x_j * s_j with one scalar per term and limb, both polynomials
// (blockIdx.z).  Bound by bytes: every term is read once and the sum written
// once, four terms of 16 bytes in flight per thread.  A product and a sum per
// term, each a pass of its own, moved five polynomials where this moves one (the
// Chebyshev sums of a bootstrap took 1.9 of 25.4 ms, now 0.6).
template <class S>
__global__ void __launch_bounds__(kThreads)
linear_kernel(const __grid_constant__ LinearArgs a, const __grid_constant__ LimbList list,
              const DevModulus* __restrict__ mods, uint32_t n) {
  const int      m = list.limb[blockIdx.y], p = blockIdx.z;
  const uint32_t i = blockIdx.x * kThreads + threadIdx.x;  // pair of coefficients
  if (i >= n / 2) return;
  const DevModulus      md = mods[m];
  const typename S::Mod sm(md);
  const size_t          off = (size_t)m * n;
  S                     s0, s1;
  s0.zero();
  s1.zero();
#pragma unroll 1
  for (int base = 0; base < a.terms; base += 4) {
    ulonglong2 x[4];
#pragma unroll
    for (int u = 0; u < 4; u++)
      x[u] = base + u < a.terms ? load2(a.x[base + u][p] + off, i) : make_ulonglong2(0, 0);
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const typename S::Word w = S::word(a.scalar[base + u][m]);
      s0.mac(S::word(x[u].x), w, sm);
      s1.mac(S::word(x[u].y), w, sm);
    }
  }
  const u64 add = p == 0 ? a.constant[m] : 0;
  reinterpret_cast<ulonglong2*>(a.out[p] + off)[i] =
      make_ulonglong2(add_mod(s0.template value<false>(sm, md), add, md.q),
                      add_mod(s1.template value<false>(sm, md), add, md.q));
}

// The limbs of an extended polynomial by the arithmetic of their primes, one
// launch each: integers first, then double precision.  A dozen limbs and fewer
// are not worth a launch of their own (2 to 3 us): the integer kernels take them.
std::array<LimbList, 2> limb_lists(Context* c, int level, int special, uint64_t skip_mask) {
  std::array<LimbList, 2> lists{};
  for (int m = 0; m < level + special; m++) {
    if (m < 64 && ((skip_mask >> m) & 1)) continue;
    LimbList& l = lists[c->ntt_float[m < level ? m : c->L + (m - level)]];
    l.limb[l.count++] = (uint8_t)m;
  }
  lists[1].is_float = true;
  if (lists[1].count <= 12 && lists[0].count > 0) {
    for (int i = 0; i < lists[1].count; i++) lists[0].limb[lists[0].count++] = lists[1].limb[i];
    lists[1].count = 0;
  }
  return lists;
}

template <typename F>
void with_sum(Context* c, const LimbList& list, F f) {
  if (list.is_float) f(SumFp());
  else if (c->primes_below_2_60) f(SumHalves());
  else f(SumWide());
}

}  // namespace

void launch_inner_product(const InnerArgs& args) {
  Context* c     = ctx();
  int      limbs = args.level + c->K;
  FHERT_ASSERT(args.parts >= 1 && args.parts <= kMaxParts, "unsupported digit count");
  DagScope dag(DAG_INNER_PRODUCT);
  if (dag.live) {
    const size_t n = c->N, w = n * sizeof(u64);
    for (int m = 0; m < limbs; m++) {
      if (m < 64 && ((args.skip_mask >> m) & 1)) continue;
      const bool   is_q  = m < args.level;
      const size_t e_off = (size_t)(is_q ? m : args.ext_p_limb + (m - args.level)) * n;
      const size_t k_off = (size_t)(is_q ? m : args.key_p_limb + (m - args.level)) * n;
      const size_t d_off = (size_t)(is_q ? m : args.acc_p_limb + (m - args.level)) * n;
      const int    own   = (args.in != nullptr && is_q) ? m / args.alpha : -1;
      for (int j = 0; j < args.parts; j++) {
        dag.set.read(j == own ? args.in + (size_t)m * n : args.ext_ptr[j] + e_off, w);
        dag.set.read(args.key0[j] + k_off, w);
        if (args.acc1 != nullptr) dag.set.read(args.key1[j] + k_off, w);
      }
      dag.set.write(args.acc0 + d_off, w);
      if (args.acc1 != nullptr) dag.set.write(args.acc1 + d_off, w);
      if (args.add[0] != nullptr && is_q)
        for (const u64* add : args.add) dag.set.read(add + d_off, w);
    }
  }
  dag.commit();
  prof_before(KID_INNER_PRODUCT);
  const unsigned x = (c->N + 4 * kThreads - 1) / (4 * kThreads);
  for (const LimbList& list : limb_lists(c, args.level, c->K, args.skip_mask)) {
    if (list.count == 0) continue;
    const dim3 g(x, list.count);
    auto go = [&](auto sum, auto two) {
      typedef decltype(sum) S;
      constexpr bool        TWO = decltype(two)::value;
      auto run = [&](auto kernel) {
        launch(kernel, g, kThreads, 0, c->stream, args, list, c->L, c->d_mod, c->N);
      };
      if (args.parts == 1) run(inner_product_kernel<TWO, S, 1, true>);
      else if (args.parts == 2) run(inner_product_kernel<TWO, S, 2, true>);
      else if (args.parts == 3) run(inner_product_kernel<TWO, S, 3, true>);
      else if (args.parts == 4) run(inner_product_kernel<TWO, S, 4, true>);
      else run(inner_product_kernel<TWO, S, 2, false>);
    };
    with_sum(c, list, [&](auto sum) {
      if (args.acc1 != nullptr) go(sum, std::true_type());
      else go(sum, std::false_type());
    });
    c->launches++;
  }
  prof_after(KID_INNER_PRODUCT, limbs);
  CUDA_CHECK(cudaGetLastError());
}

void launch_keys_product(const KeysArgs& args) {
  Context* c     = ctx();
  int      limbs = args.level + c->K;
  FHERT_ASSERT(args.count >= 1 && args.count <= kMaxKeys && args.parts >= 1 && args.parts <= kMaxParts,
               "unsupported set of rotations");
  DagScope dag(DAG_INNER_PRODUCT);
  if (dag.live) {
    const size_t w = (size_t)limbs * c->N * sizeof(u64);
    for (int j = 0; j < args.parts; j++) dag.set.read(args.digits + (size_t)j * args.digit_stride, w);
    dag.set.read(args.in, (size_t)args.level * c->N * sizeof(u64));
    if (args.c0) dag.set.read(args.c0, args.p_mod_q ? (size_t)args.level * c->N * sizeof(u64) : w);
    for (int r = 0; r < args.count; r++)
      for (int p = 0; p < 2; p++) {
        const u64* to = args.out + (size_t)r * args.out_stride + (size_t)p * args.poly_stride;
        if (args.accumulate) dag.set.read(to, w);
        dag.set.write(to, w);
      }
  }
  dag.commit();
  prof_before(KID_INNER_PRODUCT);
  const unsigned x = (c->N + kTile - 1) / kTile;
  for (const LimbList& list : limb_lists(c, args.level, c->K, 0)) {
    if (list.count == 0) continue;
    const dim3 g(x, list.count);
    with_sum(c, list, [&](auto sum) {
      typedef decltype(sum) S;
      auto run = [&](auto kernel) {
        launch(kernel, g, kTile / 2, 0, c->stream, args, list, c->L, c->d_mod, c->N);
      };
      if (args.parts == 1) run(keys_product_kernel<S, 1, true>);
      else if (args.parts == 2) run(keys_product_kernel<S, 2, true>);
      else if (args.parts == 3) run(keys_product_kernel<S, 3, true>);
      else if (args.parts == 4) run(keys_product_kernel<S, 4, true>);
      else run(keys_product_kernel<S, kMaxParts, false>);
    });
    c->launches++;
  }
  prof_after(KID_INNER_PRODUCT, limbs * args.count);
  CUDA_CHECK(cudaGetLastError());
}

void launch_weighted_sums(const SumsArgs& args) {
  Context* c     = ctx();
  int      limbs = args.level + c->K;
  FHERT_ASSERT(args.sums >= 1 && args.sums <= kMaxSums && args.terms <= kMaxParts,
               "unsupported set of sums");
  DagScope dag(DAG_INNER_PRODUCT);
  if (dag.live) {
    const size_t w = (size_t)limbs * c->N * sizeof(u64);
    for (int j = 0; j < args.terms; j++)
      for (int p = 0; p < 2; p++)
        dag.set.read(args.rot + (size_t)j * args.rot_stride + (size_t)p * args.poly_stride, w);
    for (int i = 0; i < args.sums; i++)
      for (int p = 0; p < 2; p++)
        dag.set.write(args.out + (size_t)i * args.out_stride + (size_t)p * args.poly_stride, w);
  }
  dag.commit();
  prof_before(KID_INNER_PRODUCT);
  const unsigned x = (c->N + kThreads - 1) / kThreads;
  for (const LimbList& list : limb_lists(c, args.level, c->K, 0)) {
    if (list.count == 0) continue;
    const dim3 g(x, list.count);
    with_sum(c, list, [&](auto sum) {
      typedef decltype(sum) S;
      auto run = [&](auto kernel) {
        launch(kernel, g, kThreads, 0, c->stream, args, list, c->L, c->d_mod, c->N);
      };
      if (args.sums == 1) run(weighted_sums_kernel<S, 1>);
      else if (args.sums == 2) run(weighted_sums_kernel<S, 2>);
      else if (args.sums == 3) run(weighted_sums_kernel<S, 3>);
      else run(weighted_sums_kernel<S, 4>);
    });
    c->launches++;
  }
  prof_after(KID_INNER_PRODUCT, limbs * args.sums);
  CUDA_CHECK(cudaGetLastError());
}

void launch_linear(const LinearArgs& args) {
  Context* c = ctx();
  FHERT_ASSERT(args.terms >= 1 && args.terms <= kMaxLinear && args.level <= kMaxLimbs / 2,
               "unsupported sum");
  DagScope dag(DAG_PER_LIMB_CONST);
  if (dag.live) {
    const size_t w = (size_t)args.level * c->N * sizeof(u64);
    for (int p = 0; p < 2; p++) {
      for (int j = 0; j < args.terms; j++) dag.set.read(args.x[j][p], w);
      dag.set.write(args.out[p], w);
    }
  }
  dag.commit();
  prof_before(KID_MUL_CONST);
  for (const LimbList& list : limb_lists(c, args.level, 0, 0)) {
    if (list.count == 0) continue;
    const dim3 g((c->N / 2 + kThreads - 1) / kThreads, list.count, 2);
    with_sum(c, list, [&](auto sum) {
      launch(linear_kernel<decltype(sum)>, g, kThreads, 0, c->stream, args, list, c->d_mod, c->N);
    });
    c->launches++;
  }
  prof_after(KID_MUL_CONST, 2 * args.level);
  CUDA_CHECK(cudaGetLastError());
}

}  // namespace fhert
