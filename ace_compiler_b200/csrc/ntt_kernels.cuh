// Device code of the negacyclic NTT / inverse NTT (kernels and butterflies).
//
// Dataflow and twiddle values follow the CPU runtime exactly
// (fhe-cmplr/rtlib/ant/util/src/ntt.c:167-241 forward, 245-330 inverse):
// forward = Cooley-Tukey, natural order in, bit-reversed order out, stage
// m = 1, 2, .., N/2 uses twiddle m + i for butterfly group i; inverse =
// Gentleman-Sande in the opposite order with N^-1 applied.  Residues written by
// the last pass are canonical, which makes them equal to the CPU runtime's.
//
// What bounds these kernels is the multiplier of a butterfly's modular product.
// A 32x32 -> 64 integer multiply-add keeps its pipe for four cycles per warp, a
// low 32-bit one for two, and a Shoup product of 64-bit words needs three of
// the former, two high halves (four cycles each) and four of the latter: 37
// cycles per warp and butterfly with everything around it.  A double-precision
// multiply-add takes two cycles and multiplies 53 bits exactly, so primes that
// fit (below 1.2 * 2^46: every scaling prime of the compiled programs) are
// transformed in floating point, 8 operations per butterfly, 17 cycles:
//   h = b*w, l = fma(b, w, -h)       the exact product as h + l
//   k = rint(h / p)                  with the reciprocal and the 1.5 * 2^52 trick
//   r = fma(-k, p, h) + l            b*w - k*p, |r| < 0.8 p, every step exact
// (registers-only loop, 12 butterflies per thread and round: 2120 against 990
// G butterflies/s, 0.25 against 0.53 us per limb of 2^16).  The products are
// integers below 2^97 in magnitude, so h + l is the product itself and the
// remainder is an exact integer; the result after the last reduction is the
// same canonical residue.  The error of k stays below 0.3 because values are
// kept below 25p: forward values grow by less than 0.8p per stage (at most 14p
// over 17 stages), in the inverse the sums double and are reduced once per
// four stages.
//
// Wider primes keep 64-bit integers:
//   * the Shoup quotient floor(b*w'/2^64) is taken from three partial products
//     (it may come out up to 2 too small, the product then lies in [0, 4q));
//   * b*w - quotient*q is one accumulation chain against -q;
//   * primes below 2^57.9 skip the per-butterfly range correction: forward
//     values grow by 4q per stage, inverse sums double over the four stages of
//     a register round and are brought back below 4q after it.  The 60-bit
//     primes correct per butterfly (range [0, 8q) forward, [0, 4q) inverse).
//
// A thread keeps 2^E values and does up to E stages between two exchanges:
//   whole    512 <= N <= 4096: one CTA per limb, 16 values per thread, one launch.
//   strided  first logN-8 stages: a CTA owns TC adjacent columns of the
//            (N/256) x 256 view of the limb.
//   contig   last 8 stages on contiguous 256-word blocks.
//   tiny     N < 512: shared memory, one butterfly at a time.
// The two-pass kernels use 16 values (two rounds of four stages, one exchange)
// in double precision and 8 (three rounds) in integers: with 24 instructions
// per integer butterfly, 16 values per thread measured 69 us for 48 limbs where
// 8 take 49 (straight-line code executed once per warp, and 120 registers).  A
// batch lists its integer limbs first; one grid covers both kinds, and CTAs of
// both run side by side on the two multiplier pipes.
// The inverse runs contig first, then strided.  Between the two passes the
// values stay lazy (doubles as their bit patterns).
#pragma once
#include "runtime.h"

namespace fhert {
namespace nttk {

typedef unsigned int u32;

constexpr int kContigLog   = 8;  // stages handled by the contiguous kernel
constexpr int kContigBlock = 256;
constexpr int kContigTable = kContigBlock + 16;  // twiddle entries per block
constexpr int kThreads     = 128;  // two-pass kernels
constexpr int kTinyMaxLog  = 8;  // below: no register rounds
constexpr int kWholeMaxLog = 12;

__device__ __forceinline__ u32 lo32(u64 x) { return (u32)x; }
__device__ __forceinline__ u32 hi32(u64 x) { return (u32)(x >> 32); }
__device__ __forceinline__ u64 pack64(u32 l, u32 h) {
  u64 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(l), "r"(h));
  return r;
}

__host__ __device__ constexpr int floor_log2(int v) { return v < 2 ? 0 : 1 + floor_log2(v >> 1); }

// ---- integer arithmetic ------------------------------------------------------

struct Mod {
  u64 q, nq, q2, q4;  // q, 2^64 - q, 2q, 4q
};
__device__ __forceinline__ Mod make_mod(u64 q) {
  Mod m;
  m.q  = q;
  m.nq = 0 - q;
  m.q2 = q << 1;
  m.q4 = q << 2;
  return m;
}

// addend + b*w + h*nq  (mod 2^64): two wide and four low multiply-adds
__device__ __forceinline__ u64 mul_chain(u64 addend, u64 b, u64 w, u64 h, u64 nq) {
  u64 t;
  asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(t) : "r"(lo32(b)), "r"(lo32(w)), "l"(addend));
  asm("mad.wide.u32 %0, %1, %2, %0;" : "+l"(t) : "r"(lo32(h)), "r"(lo32(nq)));
  u32 tl = lo32(t), th = hi32(t);
  asm("mad.lo.u32 %0, %1, %2, %0;" : "+r"(th) : "r"(lo32(b)), "r"(hi32(w)));
  asm("mad.lo.u32 %0, %1, %2, %0;" : "+r"(th) : "r"(hi32(b)), "r"(lo32(w)));
  asm("mad.lo.u32 %0, %1, %2, %0;" : "+r"(th) : "r"(lo32(h)), "r"(hi32(nq)));
  asm("mad.lo.u32 %0, %1, %2, %0;" : "+r"(th) : "r"(hi32(h)), "r"(lo32(nq)));
  return pack64(tl, th);
}

// b*w mod q for any 64-bit b, result in [0, 4q)
__device__ __forceinline__ u64 shoup4(u64 b, const Twiddle t, const Mod m) {
  return mul_chain(0, b, t.w, mulhi_under(b, t.wp), m.nq);
}

__device__ __forceinline__ u64 csub(u64 v, u64 bound) { return v >= bound ? v - bound : v; }

// [0, 4q) -> [0, q)
__device__ __forceinline__ u64 canon_4q(u64 v, const Mod m) { return csub(csub(v, m.q2), m.q); }

// any 64-bit v -> [0, q); r = floor(2^64 / q)
__device__ __forceinline__ u64 canon_any(u64 v, const Mod m, u64 r) {
  u64 e = mulhi_under(v, r);  // floor(v/q) - {0..3}
  u64 t;
  asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(t) : "r"(lo32(e)), "r"(lo32(m.nq)), "l"(v));
  u32 th = hi32(t);
  asm("mad.lo.u32 %0, %1, %2, %0;" : "+r"(th) : "r"(lo32(e)), "r"(hi32(m.nq)));
  asm("mad.lo.u32 %0, %1, %2, %0;" : "+r"(th) : "r"(hi32(e)), "r"(lo32(m.nq)));
  return canon_4q(pack64(lo32(t), th), m);
}

__device__ __forceinline__ u64 add_canon(u64 a, u64 b, u64 q) { return csub(a + b, q); }

__device__ __forceinline__ Twiddle ld_tw(const Twiddle* p) {
  ulonglong2 v = __ldg(reinterpret_cast<const ulonglong2*>(p));
  Twiddle    t;
  t.w  = v.x;
  t.wp = v.y;
  return t;
}

// ---- work fused into a forward transform (all optional) ------------------------
//
// Prologue of the first pass.
//   kind 1, the lift of a rescale (rns_poly.c:351-366): the source limb holds
//     residues modulo q_last in coefficient form; the value that enters the
//     transform under prime i is switch_modulus(v, q_last -> q_i) * mul[i]
//   kind 3, the lift of a rescale that follows a ModDown at once: the dropped limb
//     is y = last_x - last_conv (both multiples of P^-1 already), the source limb
//     the converted special limbs under prime i, also times P^-1; enters
//     (switch_modulus(y) + source) * mul[i], with y and source doubled for the
//     rescale of twice the polynomial.  One forward transform per limb then
//     serves both steps.
//   kind 2, a message polynomial (crt.c:1153-1221): signed 64-bit integers,
//     negatives also as kMax64 + v; their residues, times mul[i] when given
struct NttPro {
  int            kind = 0;
  const Twiddle* mul  = nullptr;  // [prime]
  const u64*     mod  = nullptr;  // [prime] q_last mod q_i
  u64            q_last = 0;
  Ptr2           last_x{{nullptr, nullptr}};
  Ptr2           last_conv{{nullptr, nullptr}};
  bool           twice = false;
};
// a message coefficient modulo q; r = floor(2^64 / q)   (modular.h:278-280)
__device__ __forceinline__ u64 message_residue(u64 v, const Mod m, u64 r) {
  constexpr long long kMax64 = (long long)((1ull << 63) - (1ull << 9)) - 1;
  long long s = (long long)v;
  if (s > (kMax64 >> 1)) s -= kMax64;
  const u64 t = canon_any(s < 0 ? 0 - (u64)s : (u64)s, m, r);
  return s < 0 && t != 0 ? m.q - t : t;
}
// Epilogue of the last pass on the canonical transform output t:
//   kind 1 (rescale, rns_poly.c:367-383):  res = aux * mul[i] + t
//   kind 2 (ModDown, rns_poly.c:293-304):  res = (aux - t) * mul[i] (+ add)
//   kind 3:  kind 2, the result then permuted, res[i] = value[perm[i]] for an
//            automorphism in NTT order.  The high bits of perm[i] depend on the
//            high bits of i alone, so blocks of 256 go to blocks of 256: a CTA
//            transforms the source blocks of its destination blocks, permutes in
//            shared memory and still writes in order (a gather of its own cost
//            23 us for 72 limbs at N = 2^16).
// aux is limb LimbRef::b of aux.p[sel bit 1]; add uses the same limb index and
// selector, a null base means no addend.
//   kind 4:  kind 2 or 3, polynomial by polynomial (NttMulti)
struct NttEpi {
  const uint32_t* perm = nullptr;
  int            kind = 0;
  const Twiddle* mul  = nullptr;  // [prime]
  Ptr2           aux{{nullptr, nullptr}};
  Ptr2           add{{nullptr, nullptr}};
};

// ---- the two arithmetics --------------------------------------------------------
//
// V: a value in registers, T: a twiddle.  load/store convert canonical words,
// bits/from_bits move lazy values between the passes.

struct ArithFp {
  typedef double V;
  typedef double T;
  static constexpr bool kFloat = true;
  double p, np, pinv;
  u64    q, rq;

  __device__ __forceinline__ explicit ArithFp(const DevModulus& d) {
    p    = (double)d.q;
    np   = -p;
    pinv = d.q_recip;
    q    = d.q;
    rq   = d.mu_hi;
  }
  static constexpr double kRound = 6755399441055744.0;  // 1.5 * 2^52
  static constexpr double kWord  = 4503599627370496.0;  // 2^52

  static __device__ __forceinline__ V from_bits(u64 v) { return __longlong_as_double((long long)v); }
  static __device__ __forceinline__ u64 bits(V v) { return (u64)__double_as_longlong(v); }
  // canonical residue (below 2^52) -> value
  static __device__ __forceinline__ V load(u64 v) {
    return __dadd_rn(__hiloint2double((int)(hi32(v) | 0x43300000u), (int)lo32(v)), -kWord);
  }
  __device__ __forceinline__ double nearest(double v) const {  // rint(v / p)
    return __dadd_rn(__fma_rn(v, pinv, kRound), -kRound);
  }
  // product of an integer below 25p with a twiddle, |result| < 0.8 p
  __device__ __forceinline__ V mul(V b, T w) const {
    double h = __dmul_rn(b, w);
    double k = nearest(h);
    double l = __fma_rn(b, w, -h);
    return __dadd_rn(__fma_rn(k, np, h), l);
  }
  __device__ __forceinline__ V reduce(V v) const { return __fma_rn(nearest(v), np, v); }
  // |v| < p -> canonical word
  __device__ __forceinline__ u64 word(V v) const {
    const long long magic = 0x4338000000000000ll;
    long long       i     = __double_as_longlong(__dadd_rn(v, kRound)) - magic;
    return (u64)(i + ((i >> 63) & (long long)q));
  }
  __device__ __forceinline__ u64 canon(V v) const { return word(reduce(v)); }

  __device__ __forceinline__ void fwd(V& a, V& b, T w) const {
    V r = mul(b, w), x = a;
    a   = __dadd_rn(x, r);
    b   = __dadd_rn(x, -r);
  }
  template <int K>
  __device__ __forceinline__ void inv(V& a, V& b, T w) const {
    V d = __dadd_rn(a, -b);
    a   = __dadd_rn(a, b);
    b   = mul(d, w);
  }
  // last inverse stage with N^-1 folded in, canonical words out
  template <int K>
  __device__ __forceinline__ void inv_last(V& a, V& b, T n_inv, T w_n) const {
    V s = __dadd_rn(a, b), d = __dadd_rn(a, -b);
    a   = from_bits(word(mul(s, n_inv)));
    b   = from_bits(word(mul(d, w_n)));
  }
  // after R inverse stages value k is a sum of 2^R inputs (k = 0) or of
  // 2^(R-1-log2 k) products: only sums of more than two need a reduction before
  // the next round
  template <int R, int K>
  __device__ __forceinline__ void settle(V& v) const {
    if (K == 0 || R - 1 - floor_log2(K) > 1) v = reduce(v);
  }
  template <int NT>
  static __device__ __forceinline__ void twiddles(T (&t)[NT], const T* p) {
    if constexpr (NT == 1) {
      t[0] = __ldg(p);
    } else {
#pragma unroll
      for (int i = 0; i < NT; i += 2) {
        double2 v = __ldg(reinterpret_cast<const double2*>(p + i));
        t[i]      = v.x;
        t[i + 1]  = v.y;
      }
    }
  }
  // stage l of a block's last four, thread g of 16
  template <int L, int NT>
  static __device__ __forceinline__ void twiddles16(T (&t)[NT], const T* block, int g) {
    if constexpr (L == 0) {
      t[0] = __ldg(block + 16 + 2 * g + 1);
    } else {
#pragma unroll
      for (int i = 0; i < NT; i += 2) {
        double2 v = __ldg(reinterpret_cast<const double2*>(block + 16 + ((NT + i) >> 1) * 32 + 2 * g));
        t[i]      = v.x;
        t[i + 1]  = v.y;
      }
    }
  }
  // a constant of the integer tables, centred like the twiddles
  __device__ __forceinline__ T constant(const Twiddle* c) const {
    double w = load(ld_tw(c).w);
    return w > 0.5 * p ? __dadd_rn(w, np) : w;
  }

  // the lift of a rescale; a dropped prime below 2^48 is centred in floating
  // point (its product with w has a quotient below 2^47), a wider one goes through words
  struct Lift {
    bool   narrow;
    u64    half, last_mod_q;
    double w, dq_last;
  };
  __device__ __forceinline__ Lift make_lift(const NttPro& pro, int prime) const {
    Lift l{};
    l.half       = pro.q_last >> 1;
    l.narrow     = (pro.q_last >> 48) == 0;
    l.last_mod_q = pro.mod[prime];
    l.w          = constant(pro.mul + prime);
    l.dq_last    = (double)pro.q_last;
    return l;
  }
  __device__ __forceinline__ V message(u64 v, bool scaled, T w) const {
    const V x = load(message_residue(v, make_mod(q), rq));
    return scaled ? mul(x, w) : x;
  }
  __device__ __forceinline__ V centred(u64 v, const Lift& l) const {
    if (l.narrow) {
      V x = load(v);
      if (v > l.half) x = __dadd_rn(x, -l.dq_last);
      return x;
    }
    const Mod m = make_mod(q);
    u64       r = canon_any(v, m, rq);
    if (v > l.half) r = r >= l.last_mod_q ? r - l.last_mod_q : r + q - l.last_mod_q;
    return load(r);
  }
  __device__ __forceinline__ V lift(u64 v, const Lift& l) const { return mul(centred(v, l), l.w); }
  __device__ __forceinline__ V lift_sum(u64 v, u64 more, bool twice, const Lift& l) const {
    const V a = load(more);
    return mul(__dadd_rn(centred(v, l), twice ? __dadd_rn(a, a) : a), l.w);
  }
  template <int EPI>
  __device__ __forceinline__ u64 epilogue(u64 t, u64 aux, T w) const {
    if (EPI == 1) return canon(__dadd_rn(mul(load(aux), w), load(t)));
    return word(mul(__dadd_rn(load(aux), -load(t)), w));
  }
};

template <bool WIDE>
struct ArithInt {
  typedef u64     V;
  typedef Twiddle T;
  static constexpr bool kFloat = false;
  Mod m;
  u64 q, rq;

  __device__ __forceinline__ explicit ArithInt(const DevModulus& d) {
    m  = make_mod(d.q);
    q  = d.q;
    rq = d.mu_hi;
  }
  static __device__ __forceinline__ V from_bits(u64 v) { return v; }
  static __device__ __forceinline__ u64 bits(V v) { return v; }
  static __device__ __forceinline__ V load(u64 v) { return v; }
  __device__ __forceinline__ u64 canon(V v) const {
    return WIDE ? canon_4q(csub(v, m.q4), m) : canon_any(v, m, rq);
  }
  __device__ __forceinline__ void fwd(V& a, V& b, const T t) const {
    u64 x = WIDE ? csub(a, m.q4) : a;
    u64 v = shoup4(b, t, m);
    a     = x + v;
    b     = x - v + m.q4;
  }
  // K: stages already done in this round; without correction sums stay below 4q << K
  template <int K>
  __device__ __forceinline__ void inv(V& a, V& b, const T t) const {
    u64 s = a + b;
    u64 d = a - b + (WIDE ? m.q4 : m.q4 << K);
    a     = WIDE ? csub(s, m.q4) : s;
    b     = shoup4(d, t, m);
  }
  template <int K>
  __device__ __forceinline__ void inv_last(V& a, V& b, const T n_inv, const T w_n) const {
    u64 s = a + b, d = a - b + (WIDE ? m.q4 : m.q4 << K);
    a     = canon_4q(shoup4(s, n_inv, m), m);
    b     = canon_4q(shoup4(d, w_n, m), m);
  }
  // after R uncorrected inverse stages value k is below 4q << R (k = 0) or
  // 4q << (R-1-log2 k): back below 4q
  template <int R, int K>
  __device__ __forceinline__ void settle(V& v) const {
    constexpr int over = K == 0 ? R : R - 1 - floor_log2(K);
    if (WIDE) return;
    if (over > 3) v = csub(v, m.q4 << 3);
    if (over > 2) v = csub(v, m.q4 << 2);
    if (over > 1) v = csub(v, m.q4 << 1);
    if (over > 0) v = csub(v, m.q4);
  }
  template <int NT>
  static __device__ __forceinline__ void twiddles(T (&t)[NT], const T* p) {
#pragma unroll
    for (int i = 0; i < NT; i++) t[i] = ld_tw(p + i);
  }
  template <int L, int NT>
  static __device__ __forceinline__ void twiddles16(T (&t)[NT], const T* block, int g) {
#pragma unroll
    for (int i = 0; i < NT; i++) t[i] = ld_tw(block + 16 + (NT + i) * 16 + g);
  }
  __device__ __forceinline__ T constant(const Twiddle* c) const { return ld_tw(c); }

  struct Lift {
    u64 half, last_mod_q;
    T   w;
  };
  __device__ __forceinline__ Lift make_lift(const NttPro& pro, int prime) const {
    return Lift{pro.q_last >> 1, pro.mod[prime], constant(pro.mul + prime)};
  }
  __device__ __forceinline__ V message(u64 v, bool scaled, const T w) const {
    const u64 r = message_residue(v, m, rq);
    return scaled ? canon_4q(shoup4(r, w, m), m) : r;
  }
  __device__ __forceinline__ V lift(u64 v, const Lift& l) const { return lift_sum(v, 0, false, l); }
  __device__ __forceinline__ V lift_sum(u64 v, u64 more, bool twice, const Lift& l) const {
    u64 r = canon_any(v, m, rq);
    if (v > l.half) r = r >= l.last_mod_q ? r - l.last_mod_q : r + q - l.last_mod_q;
    return canon_4q(shoup4(r + (twice ? 2 * more : more), l.w, m), m);
  }
  template <int EPI>
  __device__ __forceinline__ u64 epilogue(u64 t, u64 aux, const T w) const {
    if (EPI == 1) return add_canon(canon_4q(shoup4(aux, w, m), m), t, q);
    return canon_4q(shoup4(aux >= t ? aux - t : aux + q - t, w, m), m);
  }
};

// a * b mod q on the pipe the prime allows, canonical
struct Product {
  const DevModulus& m;
  ArithFp           fp;
  __device__ __forceinline__ explicit Product(const DevModulus& md) : m(md), fp(md) {}
  __device__ __forceinline__ u64 operator()(u64 a, u64 b) const {
    return m.kind == kNttFloat ? fp.word(fp.mul(ArithFp::load(a), ArithFp::load(b))) : mul_mod(a, b, m);
  }
};

// ---- register rounds --------------------------------------------------------------
//
// A thread holds the 2^E values of an E-bit field of the index; a round does the
// stages of the R highest bits of the field.  Stage l of the round (bit E-1-l)
// has 2^l groups with one twiddle each: entries node << l .. of the tree, where
// node is the tree node of the field's subtree.

template <class A>
struct TreeTw {  // tree order
  const typename A::T* table;
  u32                  node;
  template <int L, int NT>
  __device__ __forceinline__ void get(typename A::T (&t)[NT]) const {
    A::twiddles(t, table + ((size_t)node << L));
  }
};
template <class A>
struct Lanes16Tw {  // last four stages of a block, laid out for 16 lanes
  const typename A::T* block;
  int                  t;
  template <int L, int NT>
  __device__ __forceinline__ void get(typename A::T (&tw)[NT]) const {
    A::template twiddles16<L>(tw, block, t);
  }
};
struct Lanes32Tw {  // last three stages of a block of integers, laid out for 32 lanes
  const Twiddle* block;
  int            lane;
  template <int L, int NT>
  __device__ __forceinline__ void get(Twiddle (&tw)[NT]) const {
#pragma unroll
    for (int i = 0; i < NT; i++) tw[i] = ld_tw(block + 32 + ((1 << L) - 1 + i) * 32 + lane);
  }
};

// stages [L, R) of a round
template <class A, int E, int R, int L, class TW>
__device__ __forceinline__ void fwd_stages(typename A::V (&x)[1 << E], const TW& tw, const A& ar) {
  if constexpr (L < R) {
    constexpr int bit = E - 1 - L, groups = 1 << L;
    typename A::T t[groups];
    tw.template get<L>(t);
#pragma unroll
    for (int hp = 0; hp < groups; hp++)
#pragma unroll
      for (int lp = 0; lp < (1 << bit); lp++) {
        const int lo = (hp << (bit + 1)) | lp;
        ar.fwd(x[lo], x[lo | (1 << bit)], t[hp]);
      }
    fwd_stages<A, E, R, L + 1, TW>(x, tw, ar);
  }
}

// LAST: the round that reaches the first stage of the transform
template <class A, int E, int R, int L, bool LAST, class TW>
__device__ __forceinline__ void inv_stages(typename A::V (&x)[1 << E], const TW& tw, const A& ar,
                                           const Twiddle* fin) {
  if constexpr (L >= 0) {
    constexpr int bit = E - 1 - L, groups = 1 << L, done = R - 1 - L;
    if constexpr (LAST && L == 0) {
      const typename A::T n_inv = ar.constant(fin), w_n = ar.constant(fin + 1);
#pragma unroll
      for (int lp = 0; lp < (1 << bit); lp++)
        ar.template inv_last<done>(x[lp], x[lp | (1 << bit)], n_inv, w_n);
    } else {
      typename A::T t[groups];
      tw.template get<L>(t);
#pragma unroll
      for (int hp = 0; hp < groups; hp++)
#pragma unroll
        for (int lp = 0; lp < (1 << bit); lp++) {
          const int lo = (hp << (bit + 1)) | lp;
          ar.template inv<done>(x[lo], x[lo | (1 << bit)], t[hp]);
        }
    }
    inv_stages<A, E, R, L - 1, LAST, TW>(x, tw, ar, fin);
  }
}

template <class A, int E, int R, int I = 0>
__device__ __forceinline__ void settle_all(typename A::V (&x)[1 << E], const A& ar) {
  if constexpr (I < (1 << E)) {
    ar.template settle<R, (I >> (E - R))>(x[I]);
    settle_all<A, E, R, I + 1>(x, ar);
  }
}

// ---- contiguous 256-point blocks (global stages logN-8 .. logN-1) ---------------
//
// 16 lanes (16 values each): word (row r, column c) of the 16 x 16 view of the
// block sits at column c ^ r of its row: rows and columns are then both read and
// written without bank conflicts.
//   by_row: thread t touches column t of every row e (coalesced order e*16 + t)
//   by_col: thread t touches row t, columns e        (contiguous order t*16 + e)

__device__ __forceinline__ int by_row(int t, int e) { return e * 16 + (t ^ e); }
__device__ __forceinline__ int by_col(int t, int e) { return t * 16 + (e ^ t); }

// x holds e*16 + t (lazy) on entry; leaves canonical words in shared memory
template <class A>
__device__ __forceinline__ void contig16_fwd(typename A::V (&x)[16], u64* sb, int t,
                                             const typename A::T* table, const A& ar) {
  fwd_stages<A, 4, 4, 0>(x, TreeTw<A>{table, 1u}, ar);
#pragma unroll
  for (int e = 0; e < 16; e++) sb[by_row(t, e)] = A::bits(x[e]);
  __syncwarp();
#pragma unroll
  for (int e = 0; e < 16; e++) x[e] = A::from_bits(sb[by_col(t, e)]);
  fwd_stages<A, 4, 4, 0>(x, Lanes16Tw<A>{table, t}, ar);
#pragma unroll
  for (int e = 0; e < 16; e++) sb[by_col(t, e)] = ar.canon(x[e]);
  __syncwarp();
}

// canonical words in shared memory on entry; x holds e*16 + t (lazy) on exit
template <class A>
__device__ __forceinline__ void contig16_inv(typename A::V (&x)[16], u64* sb, int t,
                                             const typename A::T* table, const A& ar) {
#pragma unroll
  for (int e = 0; e < 16; e++) x[e] = A::load(sb[by_col(t, e)]);
  inv_stages<A, 4, 4, 3, false>(x, Lanes16Tw<A>{table, t}, ar, nullptr);
  settle_all<A, 4, 4>(x, ar);
#pragma unroll
  for (int e = 0; e < 16; e++) sb[by_col(t, e)] = A::bits(x[e]);
  __syncwarp();
#pragma unroll
  for (int e = 0; e < 16; e++) x[e] = A::from_bits(sb[by_row(t, e)]);
  inv_stages<A, 4, 4, 3, false>(x, TreeTw<A>{table, 1u}, ar, nullptr);
  settle_all<A, 4, 4>(x, ar);
}

// what becomes of transform word `v` of a limb with an epilogue
template <class A, int EPI>
__device__ __forceinline__ u64 finish_word(u64 v, int i, const u64* aux, const u64* add,
                                           const typename A::T& emul, const A& ar) {
  if (EPI != 0) {
    v = ar.template epilogue<EPI>(v, aux[i], emul);
    if (EPI >= 2 && add != nullptr) v = add_canon(v, add[i], ar.q);
  }
  return v;
}

// place of word i of a block in its swizzled shared memory (16 lanes)
__device__ __forceinline__ int place16(int i) { return i ^ ((i >> 4) & 15); }

template <class A, int EPI>
__device__ __forceinline__ void write_block16(u64* dst, u64* sb, int t, const u64* aux, const u64* add,
                                              const typename A::T& emul, const A& ar,
                                              const uint32_t* perm) {
#pragma unroll
  for (int e = 0; e < 16; e++) {
    const u64 v = finish_word<A, EPI>(sb[by_row(t, e)], e * 16 + t, aux, add, emul, ar);
    if (EPI >= 3 && perm != nullptr) sb[by_row(t, e)] = v;
    else dst[e * 16 + t] = v;
  }
  if (EPI >= 3 && perm != nullptr) {
    __syncwarp();
#pragma unroll
    for (int e = 0; e < 16; e++)
      dst[e * 16 + t] = sb[place16((int)__ldg(perm + e * 16 + t) & (kContigBlock - 1))];
  }
}

// 32 lanes (8 values each), rounds of 2, 3 and 3 stages with the index patterns
// e*32 + g, (b2 | e*8), g*8 + e.  The swizzle is a permutation inside each
// aligned 16-word group that keeps every half-warp on 16 distinct 8-byte banks
// for all three; it is linear over XOR, so with the block's shared memory
// aligned to its size the addresses of one thread differ by constants.
__host__ __device__ constexpr int swz(int i) {
  return i ^ ((i >> 4) & 1) ^ (((i >> 5) & 1) << 1) ^ (((i >> 6) & 1) * 12);
}
__device__ __forceinline__ u64 lds64(u32 addr) {
  u64 v;
  asm volatile("ld.shared.u64 %0, [%1];" : "=l"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void sts64(u32 addr, u64 v) {
  asm volatile("st.shared.u64 [%0], %1;" ::"r"(addr), "l"(v) : "memory");
}

template <bool INV, int EPI, class A>
__device__ __forceinline__ void contig_int(const u64* src, u64* dst, u32 sbase, int g,
                                           const Twiddle* table, const A& ar, const u64* aux,
                                           const u64* add, const Twiddle* emul,
                                           const uint32_t* perm) {
  u64       x[8];
  const int b2 = ((g >> 3) << 6) | (g & 7);
  const u32 a1 = sbase ^ (u32)(swz(g) << 3);
  const u32 a2 = sbase ^ (u32)(swz(b2) << 3);
  const u32 a3 = sbase ^ (u32)(swz(g << 3) << 3);
  const TreeTw<A>  first{table, 1u}, second{table, 4u + (u32)(g >> 3)};
  const Lanes32Tw  third{table, g};
  if constexpr (!INV) {
#pragma unroll
    for (int e = 0; e < 8; e++) x[e] = src[e * 32 + g];
    fwd_stages<A, 3, 2, 0>(x, first, ar);
#pragma unroll
    for (int e = 0; e < 8; e++) sts64(a1 ^ (u32)(swz(e << 5) << 3), x[e]);
    __syncwarp();
#pragma unroll
    for (int e = 0; e < 8; e++) x[e] = lds64(a2 ^ (u32)(swz(e << 3) << 3));
    fwd_stages<A, 3, 3, 0>(x, second, ar);
#pragma unroll
    for (int e = 0; e < 8; e++) sts64(a2 ^ (u32)(swz(e << 3) << 3), x[e]);
    __syncwarp();
#pragma unroll
    for (int e = 0; e < 8; e++) x[e] = lds64(a3 ^ (u32)(swz(e) << 3));
    fwd_stages<A, 3, 3, 0>(x, third, ar);
#pragma unroll
    for (int e = 0; e < 8; e++) sts64(a3 ^ (u32)(swz(e) << 3), ar.canon(x[e]));
    __syncwarp();
    typename A::T w{};
    if (EPI != 0) w = ar.constant(emul);
#pragma unroll
    for (int e = 0; e < 8; e++) {
      const u32 at = a1 ^ (u32)(swz(e << 5) << 3);
      const u64 v  = finish_word<A, EPI>(lds64(at), e * 32 + g, aux, add, w, ar);
      if (EPI >= 3 && perm != nullptr) sts64(at, v);
      else dst[e * 32 + g] = v;
    }
    if (EPI >= 3 && perm != nullptr) {
      __syncwarp();
#pragma unroll
      for (int e = 0; e < 8; e++) {
        const int s = (int)__ldg(perm + e * 32 + g) & (kContigBlock - 1);
        dst[e * 32 + g] = lds64(sbase ^ (u32)(swz(s) << 3));
      }
    }
  } else {
#pragma unroll
    for (int e = 0; e < 8; e++) sts64(a1 ^ (u32)(swz(e << 5) << 3), src[e * 32 + g]);
    __syncwarp();
#pragma unroll
    for (int e = 0; e < 8; e++) x[e] = lds64(a3 ^ (u32)(swz(e) << 3));
    inv_stages<A, 3, 3, 2, false>(x, third, ar, nullptr);
    settle_all<A, 3, 3>(x, ar);
#pragma unroll
    for (int e = 0; e < 8; e++) sts64(a3 ^ (u32)(swz(e) << 3), x[e]);
    __syncwarp();
#pragma unroll
    for (int e = 0; e < 8; e++) x[e] = lds64(a2 ^ (u32)(swz(e << 3) << 3));
    inv_stages<A, 3, 3, 2, false>(x, second, ar, nullptr);
    settle_all<A, 3, 3>(x, ar);
#pragma unroll
    for (int e = 0; e < 8; e++) sts64(a2 ^ (u32)(swz(e << 3) << 3), x[e]);
    __syncwarp();
#pragma unroll
    for (int e = 0; e < 8; e++) x[e] = lds64(a1 ^ (u32)(swz(e << 5) << 3));
    inv_stages<A, 3, 2, 1, false>(x, first, ar, nullptr);
    settle_all<A, 3, 2>(x, ar);
#pragma unroll
    for (int e = 0; e < 8; e++) dst[e * 32 + g] = x[e];
  }
}

template <bool INV, int EPI>
__device__ __forceinline__ void contig_float(const u64* src, u64* dst, u64* sb, int t,
                                             const double* table, const ArithFp& ar, const u64* aux,
                                             const u64* add, const Twiddle* emul,
                                             const uint32_t* perm) {
  double x[16];
  if constexpr (!INV) {
#pragma unroll
    for (int e = 0; e < 16; e++) x[e] = ArithFp::from_bits(src[e * 16 + t]);
    contig16_fwd<ArithFp>(x, sb, t, table, ar);
    double w = 0;
    if (EPI != 0) w = ar.constant(emul);
    write_block16<ArithFp, EPI>(dst, sb, t, aux, add, w, ar, perm);
  } else {
#pragma unroll
    for (int e = 0; e < 16; e++) sb[by_row(t, e)] = src[e * 16 + t];
    __syncwarp();
    contig16_inv<ArithFp>(x, sb, t, table, ar);
#pragma unroll
    for (int e = 0; e < 16; e++) dst[e * 16 + t] = ArithFp::bits(x[e]);
  }
}

// CTA -> limb of the batch and tile of the limb.  Limbs [0, n_int) of the batch
// are transformed in integers, 2^log_int tiles each, the others in double
// precision, 2^log_float tiles each.
struct TileMap {
  u32 n_int, log_int, log_float;
};
__device__ __forceinline__ bool locate(const TileMap& map, u32& limb, u32& tile) {
  const u32 ints = map.n_int << map.log_int;
  if (blockIdx.x < ints) {
    limb = blockIdx.x >> map.log_int;
    tile = blockIdx.x & ((1u << map.log_int) - 1);
    return true;
  }
  const u32 b = blockIdx.x - ints;
  limb = map.n_int + (b >> map.log_float);
  tile = b & ((1u << map.log_float) - 1);
  return false;
}

template <int EPI>
struct MultiArg {};
template <>
struct MultiArg<4> {
  NttMulti m;
};

template <bool INV, int EPI>
__global__ void __launch_bounds__(kThreads, 6)
ntt_contig_kernel(Ptr2 in, Ptr2 out, const __grid_constant__ LimbBatch batch, TileMap map,
                  const Twiddle* __restrict__ tables, const DevModulus* __restrict__ mods, uint32_t n,
                  int logn, NttEpi epi, const __grid_constant__ MultiArg<EPI> multi) {
  // 16 KiB for the blocks and up to 2 KiB to align them
  __shared__ u64 sm[kThreads / 16 * kContigBlock + kContigBlock];
  u32              limb, tile;
  const bool       is_int = locate(map, limb, tile);
  const LimbRef    lr     = batch.limb[limb];
  const DevModulus dm     = mods[lr.prime];
  const int        s1     = logn - kContigLog;
  const Twiddle*   tab    = tables + (size_t)lr.prime * table_entries(logn);
  const int        per    = is_int ? 32 : 16;  // lanes per block
  const int        slot = threadIdx.x / per, t = threadIdx.x & (per - 1);
  const u32        to     = tile * (kThreads / per) + slot;  // block of the result
  const uint32_t*  perm   = nullptr;
  if (EPI == 3) perm = epi.perm;
  if constexpr (EPI == 4) perm = multi.m.perm[lr.sel];
  if (perm != nullptr) perm += (size_t)to * kContigBlock;
  const u32        blk    = EPI >= 3 && perm != nullptr ? __ldg(perm) / kContigBlock : to;
  const size_t     off    = (size_t)blk * kContigBlock;
  const bool       two    = EPI != 4;
  const u64*       src    = (two && (lr.sel & 1) ? in.p[1] : in.p[0]) + (size_t)lr.a * n + off;
  u64*             dst    = two && (lr.sel & 4) ? out.p[1] : out.p[0];
  if constexpr (EPI == 4) dst = multi.m.out[lr.sel];
  dst += (size_t)lr.dst * n + (size_t)to * kContigBlock;
  const u64* aux = nullptr;
  const u64* add = nullptr;
  if (EPI != 0) {
    const size_t aoff = (size_t)lr.b * n + off;
    aux = (two && (lr.sel & 2) ? epi.aux.p[1] : epi.aux.p[0]) + aoff;
    add = (lr.sel & 2) ? epi.add.p[1] : epi.add.p[0];
    if constexpr (EPI == 4) add = multi.m.add[lr.sel];
    if (add != nullptr) add += two ? aoff : (size_t)lr.dst * n + off;
  }
  const Twiddle* emul  = EPI != 0 ? epi.mul + lr.prime : nullptr;
  const size_t   entry = ((size_t)1 << s1) + (size_t)blk * kContigTable;
  if (is_int) {
    const u32 sbase = (((u32)__cvta_generic_to_shared(sm) + 2047u) & ~2047u) + (u32)slot * 2048u;
    if (dm.kind == kNttNarrow)
      contig_int<INV, EPI>(src, dst, sbase, t, tab + entry, ArithInt<false>(dm), aux, add, emul,
                           perm);
    else
      contig_int<INV, EPI>(src, dst, sbase, t, tab + entry, ArithInt<true>(dm), aux, add, emul,
                           perm);
  } else {
    contig_float<INV, EPI>(src, dst, sm + slot * kContigBlock, t,
                           reinterpret_cast<const double*>(tab) + entry, ArithFp(dm), aux, add, emul,
                           perm);
  }
}

// ---- strided columns (global stages 0 .. logN-9) ---------------------------
//
// S1 = logN - 8 stages on 2^S1 rows; TC columns per CTA; threads = TC * 2^(S1-E).
// The first forward round does the odd S1 % E stages (or E), the others E each;
// the inverse runs the same rounds backwards.

__host__ __device__ constexpr int first_round(int s, int e) { return s % e == 0 ? e : s % e; }

// row r, column c of the tile; rows 2^E apart would meet in the same banks when
// a tile row is shorter than 128 bytes
template <int E, int TC>
__device__ __forceinline__ int tile_at(int row, int c) {
  constexpr int spread = TC < 16 ? 16 / TC - 1 : 0;
  return ((row ^ ((row >> E) & spread)) * TC) | c;
}

template <class A, int E, int S, int TC, int L0>
__device__ __forceinline__ void strided_fwd(typename A::V (&x)[1 << E], u64* sm, int g, int c,
                                            const typename A::T* table, const A& ar) {
  constexpr int R    = L0 == 0 ? first_round(S, E) : E;
  constexpr int LP   = L0 == 0 ? S - E : S - L0 - E;
  const int     base = ((g >> LP) << (LP + E)) | (g & ((1 << LP) - 1));
  if constexpr (L0 != 0) {
    __syncthreads();
#pragma unroll
    for (int e = 0; e < (1 << E); e++) x[e] = A::from_bits(sm[tile_at<E, TC>(base | (e << LP), c)]);
  }
  fwd_stages<A, E, R, 0>(x, TreeTw<A>{table, (1u << L0) + ((u32)base >> (LP + E))}, ar);
  if constexpr (L0 + R < S) {
    if constexpr (L0 != 0) __syncthreads();
#pragma unroll
    for (int e = 0; e < (1 << E); e++) sm[tile_at<E, TC>(base | (e << LP), c)] = A::bits(x[e]);
    strided_fwd<A, E, S, TC, L0 + R>(x, sm, g, c, table, ar);
  }
}

// HI: stages [0, HI) are still to do
template <class A, int E, int S, int TC, int HI>
__device__ __forceinline__ void strided_inv(typename A::V (&x)[1 << E], u64* sm, int g, int c,
                                            const typename A::T* table, const A& ar,
                                            const Twiddle* fin) {
  constexpr bool LAST = HI == first_round(S, E);
  constexpr int  R    = LAST ? HI : E;
  constexpr int  L0   = HI - R;
  constexpr int  LP   = LAST ? S - E : S - L0 - E;
  const int      base = ((g >> LP) << (LP + E)) | (g & ((1 << LP) - 1));
  if constexpr (HI != S) {
    __syncthreads();
#pragma unroll
    for (int e = 0; e < (1 << E); e++) x[e] = A::from_bits(sm[tile_at<E, TC>(base | (e << LP), c)]);
  }
  inv_stages<A, E, R, R - 1, LAST>(x, TreeTw<A>{table, (1u << L0) + ((u32)base >> (LP + E))}, ar, fin);
  if constexpr (!LAST) {
    settle_all<A, E, R>(x, ar);
    if constexpr (HI != S) __syncthreads();
#pragma unroll
    for (int e = 0; e < (1 << E); e++) sm[tile_at<E, TC>(base | (e << LP), c)] = A::bits(x[e]);
    strided_inv<A, E, S, TC, L0>(x, sm, g, c, table, ar, fin);
  }
}

// (the prologue is a template parameter: its code in a kernel that does not use
// it cost 2 us a launch)
// at(e): where in the limb value e stands; last: the dropped limb's pair (kind 3)
struct LastLimb {
  const u64* x    = nullptr;
  const u64* conv = nullptr;
};
template <class A, int E, int PRO, class At>
__device__ __forceinline__ void load_values(typename A::V (&x)[1 << E], const u64 (&v)[1 << E],
                                            const A& ar, const NttPro& pro, int prime,
                                            const LastLimb& last, At at) {
  if constexpr (PRO == 3) {
    const typename A::Lift lift = ar.make_lift(pro, prime);
    const u64              ql   = pro.q_last;
#pragma unroll
    for (int e = 0; e < (1 << E); e++) {
      u64 y = last.x[at(e)], s = last.conv[at(e)];
      y = y >= s ? y - s : y + ql - s;
      if (pro.twice) y = csub(2 * y, ql);
      x[e] = ar.lift_sum(y, v[e], pro.twice, lift);
    }
  } else if constexpr (PRO == 1) {
    const typename A::Lift lift = ar.make_lift(pro, prime);
#pragma unroll
    for (int e = 0; e < (1 << E); e++) x[e] = ar.lift(v[e], lift);
  } else if constexpr (PRO == 2) {
    const bool          scaled = pro.mul != nullptr;
    const typename A::T w      = scaled ? ar.constant(pro.mul + prime) : typename A::T{};
#pragma unroll
    for (int e = 0; e < (1 << E); e++) x[e] = ar.message(v[e], scaled, w);
  } else {
#pragma unroll
    for (int e = 0; e < (1 << E); e++) x[e] = A::load(v[e]);
  }
}

template <bool INV, int PRO, int E, int S1, int TC, class A>
__device__ __forceinline__ void strided_body(const u64* src, u64* dst, u64* sm, const Twiddle* table,
                                             const A& ar, const Twiddle* fin, const NttPro& pro,
                                             int prime, LastLimb last) {
  const typename A::T* tw = reinterpret_cast<const typename A::T*>(table);
  const int            c = threadIdx.x % TC, g = threadIdx.x / TC;
  typename A::V        x[1 << E];
  // the field of the first and of the last round: top E row bits, low E row bits
  constexpr int top = S1 - E;
  const int     at_top = g, at_low = g << E;
  src += c;
  dst += c;
  if constexpr (!INV) {
    auto at = [&](int e) { return (size_t)(at_top | (e << top)) << kContigLog; };
    u64  v[1 << E];
#pragma unroll
    for (int e = 0; e < (1 << E); e++) v[e] = src[at(e)];
    last.x += c;
    last.conv += c;
    load_values<A, E, PRO>(x, v, ar, pro, prime, last, at);
    strided_fwd<A, E, S1, TC, 0>(x, sm, g, c, tw, ar);
#pragma unroll
    for (int e = 0; e < (1 << E); e++) dst[(size_t)(at_low | e) << kContigLog] = A::bits(x[e]);
  } else {
#pragma unroll
    for (int e = 0; e < (1 << E); e++) x[e] = A::from_bits(src[(size_t)(at_low | e) << kContigLog]);
    strided_inv<A, E, S1, TC, S1>(x, sm, g, c, tw, ar, fin);
#pragma unroll
    for (int e = 0; e < (1 << E); e++) dst[(size_t)(at_top | (e << top)) << kContigLog] = A::bits(x[e]);
  }
}

// columns per CTA: kThreads threads at every ring degree
__host__ __device__ constexpr int tile_columns(int s1, int e) { return kThreads >> (s1 - e); }

template <bool INV, int PRO, int S1>
__global__ void __launch_bounds__(kThreads, 7)
ntt_strided_kernel(Ptr2 in, Ptr2 out, const __grid_constant__ LimbBatch batch, TileMap map,
                   const Twiddle* __restrict__ tables, const DevModulus* __restrict__ mods,
                   const Twiddle* __restrict__ inv_last, uint32_t n,
                   const __grid_constant__ NttPro pro) {
  constexpr int TI = tile_columns(S1, 3), TF = tile_columns(S1, 4);
  __shared__ u64   sm[TF << S1];
  u32              limb, tile;
  const bool       is_int = locate(map, limb, tile);
  const LimbRef    lr     = batch.limb[limb];
  const DevModulus dm     = mods[lr.prime];
  const Twiddle*   tab    = tables + (size_t)lr.prime * table_entries(S1 + kContigLog);
  const Twiddle*   fin    = inv_last + (size_t)lr.prime * 2;
  const size_t     col    = (size_t)tile * (is_int ? TI : TF);
  const u64*       src    = ((lr.sel & 1) ? in.p[1] : in.p[0]) + (size_t)lr.a * n + col;
  u64*             dst    = ((lr.sel & 4) ? out.p[1] : out.p[0]) + (size_t)lr.dst * n + col;
  LastLimb last;
  if (PRO == 3) last = LastLimb{pro.last_x.p[lr.sel & 1] + col, pro.last_conv.p[lr.sel & 1] + col};
  if (!is_int)
    strided_body<INV, PRO, 4, S1, TF>(src, dst, sm, tab, ArithFp(dm), fin, pro, lr.prime, last);
  else if (dm.kind == kNttNarrow)
    strided_body<INV, PRO, 3, S1, TI>(src, dst, sm, tab, ArithInt<false>(dm), fin, pro, lr.prime, last);
  else
    strided_body<INV, PRO, 3, S1, TI>(src, dst, sm, tab, ArithInt<true>(dm), fin, pro, lr.prime, last);
}

// ---- whole limb in one CTA (512 <= N <= 4096) ------------------------------------
//
// S1 = logN - 8 stages in one register round over the top bits, then the
// contiguous rounds; N/16 threads.

template <bool INV, int PRO, int EPI, int S1, class A>
__device__ __forceinline__ void whole_body(const u64* src, u64* dst, u64* sm, const Twiddle* table,
                                           const DevModulus& dm, const Twiddle* fin,
                                           const NttPro& pro, int prime, const u64* aux,
                                           const u64* add, const Twiddle* emul, const uint32_t* perm,
                                           const LastLimb& last) {
  constexpr int        logn = S1 + kContigLog, top = logn - 4;
  const A              ar(dm);
  const typename A::T* tree = reinterpret_cast<const typename A::T*>(table);
  const int            g = threadIdx.x, half = g >> 4, t = g & 15;
  const typename A::T* blk   = tree + ((size_t)1 << S1) + (size_t)half * kContigTable;
  u64*                 sb    = sm + half * kContigBlock;
  typename A::V        x[16];
  // word i of the limb in the swizzled view of its block
  auto at = [](int i) { return i ^ ((i >> 4) & 15); };
  if constexpr (!INV) {
    u64 v[16];
#pragma unroll
    for (int e = 0; e < 16; e++) v[e] = src[g | (e << top)];
    load_values<A, 4, PRO>(x, v, ar, pro, prime, last, [&](int e) { return g | (e << top); });
    fwd_stages<A, 4, S1, 0>(x, TreeTw<A>{tree, 1u}, ar);
#pragma unroll
    for (int e = 0; e < 16; e++) sm[at(g | (e << top))] = A::bits(x[e]);
    __syncthreads();
#pragma unroll
    for (int e = 0; e < 16; e++) x[e] = A::from_bits(sb[by_row(t, e)]);
    __syncwarp();
    contig16_fwd<A>(x, sb, t, blk, ar);
    typename A::T w{};
    if (EPI != 0) w = ar.constant(emul);
    const size_t off = (size_t)half * kContigBlock;
    if (EPI < 3 || perm == nullptr) {
      write_block16<A, EPI>(dst + off, sb, t, aux + off, add != nullptr ? add + off : nullptr, w, ar,
                            nullptr);
    } else {
#pragma unroll
      for (int e = 0; e < 16; e++)
        sb[by_row(t, e)] = finish_word<A, EPI>(sb[by_row(t, e)], (int)off + e * 16 + t, aux, add, w, ar);
      __syncthreads();
#pragma unroll
      for (int e = 0; e < 16; e++) dst[off + e * 16 + t] = sm[place16((int)__ldg(perm + off + e * 16 + t))];
    }
  } else {
    const size_t off = (size_t)half * kContigBlock;
#pragma unroll
    for (int e = 0; e < 16; e++) sb[by_row(t, e)] = src[off + e * 16 + t];
    __syncwarp();
    contig16_inv<A>(x, sb, t, blk, ar);
#pragma unroll
    for (int e = 0; e < 16; e++) sb[by_row(t, e)] = A::bits(x[e]);
    __syncthreads();
#pragma unroll
    for (int e = 0; e < 16; e++) x[e] = A::from_bits(sm[at(g | (e << top))]);
    inv_stages<A, 4, S1, S1 - 1, true>(x, TreeTw<A>{tree, 1u}, ar, fin);
#pragma unroll
    for (int e = 0; e < 16; e++) dst[g | (e << top)] = A::bits(x[e]);
  }
}

template <bool INV, int PRO, int EPI, int S1>
__global__ void __launch_bounds__(16 << S1)
ntt_whole_kernel(Ptr2 in, Ptr2 out, LimbBatch batch, const Twiddle* __restrict__ tables,
                 const DevModulus* __restrict__ mods, const Twiddle* __restrict__ inv_last,
                 const __grid_constant__ NttPro pro, NttEpi epi, const __grid_constant__ MultiArg<EPI> multi) {
  constexpr uint32_t n = (uint32_t)kContigBlock << S1;
  __shared__ u64 sm[n];
  const LimbRef    lr  = batch.limb[blockIdx.x];
  const DevModulus dm  = mods[lr.prime];
  const Twiddle*   tab = tables + (size_t)lr.prime * table_entries(S1 + kContigLog);
  const Twiddle*   fin = inv_last + (size_t)lr.prime * 2;
  const bool       two = EPI != 4;
  const u64*       src = (two && (lr.sel & 1) ? in.p[1] : in.p[0]) + (size_t)lr.a * n;
  u64*             dst = two && (lr.sel & 4) ? out.p[1] : out.p[0];
  const uint32_t*  perm = EPI == 3 ? epi.perm : nullptr;
  const u64* aux = nullptr;
  const u64* add = nullptr;
  if (EPI != 0) {
    aux = (two && (lr.sel & 2) ? epi.aux.p[1] : epi.aux.p[0]) + (size_t)lr.b * n;
    add = (lr.sel & 2) ? epi.add.p[1] : epi.add.p[0];
    if constexpr (EPI == 4) add = multi.m.add[lr.sel];
    if (add != nullptr) add += (size_t)(two ? lr.b : lr.dst) * n;
  }
  if constexpr (EPI == 4) {
    dst  = multi.m.out[lr.sel];
    perm = multi.m.perm[lr.sel];
  }
  dst += (size_t)lr.dst * n;
  const Twiddle* emul = EPI != 0 ? epi.mul + lr.prime : nullptr;
  LastLimb       last;
  if (PRO == 3) last = LastLimb{pro.last_x.p[lr.sel & 1], pro.last_conv.p[lr.sel & 1]};
  if (dm.kind == kNttFloat)
    whole_body<INV, PRO, EPI, S1, ArithFp>(src, dst, sm, tab, dm, fin, pro, lr.prime, aux, add, emul,
                                       perm, last);
  else if (dm.kind == kNttNarrow)
    whole_body<INV, PRO, EPI, S1, ArithInt<false>>(src, dst, sm, tab, dm, fin, pro, lr.prime, aux, add, emul,
                                       perm, last);
  else
    whole_body<INV, PRO, EPI, S1, ArithInt<true>>(src, dst, sm, tab, dm, fin, pro, lr.prime, aux, add, emul,
                                       perm, last);
}

// ---- tiny transforms (N < 512): one butterfly at a time --------------------------
// Always the corrected (wide) butterflies; twiddles in tree order.

template <bool INV>
__global__ void ntt_tiny_kernel(Ptr2 in, Ptr2 out, LimbBatch batch,
                                const Twiddle* __restrict__ tables,
                                const DevModulus* __restrict__ mods,
                                const Twiddle* __restrict__ inv_last, uint32_t n, int logn) {
  __shared__ u64 sm[1 << kTinyMaxLog];
  const LimbRef        lr = batch.limb[blockIdx.x];
  const ArithInt<true> ar(mods[lr.prime]);
  const Twiddle* tw  = tables + (size_t)lr.prime * table_entries(logn);
  const Twiddle* fin = inv_last + (size_t)lr.prime * 2;
  const u64*     src = ((lr.sel & 1) ? in.p[1] : in.p[0]) + (size_t)lr.a * n;
  u64*           dst = ((lr.sel & 4) ? out.p[1] : out.p[0]) + (size_t)lr.dst * n;
  for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) sm[i] = src[i];
  __syncthreads();
  for (int k = 0; k < logn; k++) {
    const int l = INV ? logn - 1 - k : k, tlog = logn - 1 - l;
    for (uint32_t bf = threadIdx.x; bf < (n >> 1); bf += blockDim.x) {
      const uint32_t i  = bf >> tlog;
      const uint32_t j1 = (i << (tlog + 1)) | (bf & ((1u << tlog) - 1));
      u64 a = sm[j1], b = sm[j1 + (1u << tlog)];
      if (!INV) ar.fwd(a, b, ld_tw(tw + (1u << l) + i));
      else if (l == 0) ar.inv_last<0>(a, b, ld_tw(fin), ld_tw(fin + 1));
      else ar.inv<0>(a, b, ld_tw(tw + (1u << l) + i));
      sm[j1]                 = a;
      sm[j1 + (1u << tlog)] = b;
    }
    __syncthreads();
  }
  for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) dst[i] = INV ? sm[i] : ar.canon(sm[i]);
}

// Tables and geometry of one transform launch.
struct NttTables {
  const Twiddle*    fwd;
  const Twiddle*    inv;
  const Twiddle*    inv_last;
  const DevModulus* mods;
  uint32_t          n;
  int               logn;
};

// n_int: how many limbs, at the front of the batch, are transformed in integers
template <bool INV, int PRO, int S1>
inline void launch_strided_t(Ptr2 in, Ptr2 out, const LimbBatch& b, int n_int, const NttTables& t,
                             cudaStream_t stream, const NttPro& pro) {
  const TileMap map{(u32)n_int, (u32)(kContigLog - floor_log2(tile_columns(S1, 3))),
                    (u32)(kContigLog - floor_log2(tile_columns(S1, 4)))};
  const int     ctas = (n_int << map.log_int) + ((b.count - n_int) << map.log_float);
  launch(ntt_strided_kernel<INV, PRO, S1>, ctas, kThreads, 0, stream, in, out, b, map,
         INV ? t.inv : t.fwd, t.mods, t.inv_last, t.n, pro);
}

template <bool INV, int PRO>
inline void launch_strided_p(Ptr2 in, Ptr2 out, const LimbBatch& b, int n_int, const NttTables& t,
                             cudaStream_t stream, const NttPro& pro) {
  switch (t.logn - kContigLog) {
    case 5: launch_strided_t<INV, PRO, 5>(in, out, b, n_int, t, stream, pro); break;
    case 6: launch_strided_t<INV, PRO, 6>(in, out, b, n_int, t, stream, pro); break;
    case 7: launch_strided_t<INV, PRO, 7>(in, out, b, n_int, t, stream, pro); break;
    case 8: launch_strided_t<INV, PRO, 8>(in, out, b, n_int, t, stream, pro); break;
    case 9: launch_strided_t<INV, PRO, 9>(in, out, b, n_int, t, stream, pro); break;
    default: FHERT_ASSERT(false, "ring degree 2^%d has no transform kernel", t.logn);
  }
}

template <bool INV>
inline void launch_strided(Ptr2 in, Ptr2 out, const LimbBatch& b, int n_int, const NttTables& t,
                           cudaStream_t stream, const NttPro& pro = NttPro()) {
  if (INV || pro.kind == 0) launch_strided_p<INV, 0>(in, out, b, n_int, t, stream, pro);
  else if (pro.kind == 1) launch_strided_p<false, 1>(in, out, b, n_int, t, stream, pro);
  else if (pro.kind == 3) launch_strided_p<false, 3>(in, out, b, n_int, t, stream, pro);
  else launch_strided_p<false, 2>(in, out, b, n_int, t, stream, pro);
}

template <bool INV>
inline void launch_contig(Ptr2 in, Ptr2 out, const LimbBatch& b, int n_int, const NttTables& t,
                          cudaStream_t stream, const NttEpi& epi = NttEpi(),
                          const NttMulti* multi = nullptr) {
  const u32      blocks = (u32)(t.logn - kContigLog);
  const TileMap  map{(u32)n_int, blocks - floor_log2(kThreads / 32), blocks - floor_log2(kThreads / 16)};
  const int      ctas = (n_int << map.log_int) + ((b.count - n_int) << map.log_float);
  const Twiddle* tab  = INV ? t.inv : t.fwd;
  if (INV || epi.kind == 0)
    launch(ntt_contig_kernel<INV, 0>, ctas, kThreads, 0, stream, in, out, b, map, tab, t.mods, t.n,
           t.logn, epi, MultiArg<0>{});
  else if (epi.kind == 1)
    launch(ntt_contig_kernel<false, 1>, ctas, kThreads, 0, stream, in, out, b, map, tab, t.mods, t.n,
           t.logn, epi, MultiArg<1>{});
  else if (epi.kind == 4)
    launch(ntt_contig_kernel<false, 4>, ctas, kThreads, 0, stream, in, out, b, map, tab, t.mods, t.n,
           t.logn, epi, MultiArg<4>{*multi});
  else if (epi.kind == 3)
    launch(ntt_contig_kernel<false, 3>, ctas, kThreads, 0, stream, in, out, b, map, tab, t.mods, t.n,
           t.logn, epi, MultiArg<3>{});
  else
    launch(ntt_contig_kernel<false, 2>, ctas, kThreads, 0, stream, in, out, b, map, tab, t.mods, t.n,
           t.logn, epi, MultiArg<2>{});
}

template <bool INV, int PRO, int EPI>
inline void launch_whole_t(Ptr2 in, Ptr2 out, const LimbBatch& b, const NttTables& t,
                           cudaStream_t stream, const NttPro& pro, const NttEpi& epi,
                           const MultiArg<EPI>& multi) {
  const Twiddle* tab = INV ? t.inv : t.fwd;
#define WHOLE_CASE(S1_)                                                                           \
  launch(ntt_whole_kernel<INV, PRO, EPI, S1_>, b.count, 16 << S1_, 0, stream, in, out, b, tab, t.mods, \
         t.inv_last, pro, epi, multi)
  switch (t.logn - kContigLog) {
    case 1: WHOLE_CASE(1); break;
    case 2: WHOLE_CASE(2); break;
    case 3: WHOLE_CASE(3); break;
    default: WHOLE_CASE(4); break;
  }
#undef WHOLE_CASE
}

template <bool INV>
inline void launch_whole(Ptr2 in, Ptr2 out, const LimbBatch& b, const NttTables& t,
                         cudaStream_t stream, const NttPro& pro = NttPro(),
                         const NttEpi& epi = NttEpi(), const NttMulti* multi = nullptr) {
  // a lift comes with a rescale's last step, a message with none
  FHERT_ASSERT(pro.kind == 0 || ((pro.kind & 1) && epi.kind == 1) || (pro.kind == 2 && epi.kind == 0),
               "no transform with prologue %d and epilogue %d", pro.kind, epi.kind);
  if (pro.kind == 1) launch_whole_t<false, 1, 1>(in, out, b, t, stream, pro, epi, MultiArg<1>{});
  else if (pro.kind == 3) launch_whole_t<false, 3, 1>(in, out, b, t, stream, pro, epi, MultiArg<1>{});
  else if (pro.kind == 2) launch_whole_t<false, 2, 0>(in, out, b, t, stream, pro, epi, MultiArg<0>{});
  else if (INV || epi.kind == 0) launch_whole_t<INV, 0, 0>(in, out, b, t, stream, pro, epi, MultiArg<0>{});
  else if (epi.kind == 3) launch_whole_t<false, 0, 3>(in, out, b, t, stream, pro, epi, MultiArg<3>{});
  else if (epi.kind == 4) launch_whole_t<false, 0, 4>(in, out, b, t, stream, pro, epi, MultiArg<4>{*multi});
  else launch_whole_t<false, 0, 2>(in, out, b, t, stream, pro, epi, MultiArg<2>{});
}

template <bool INV>
inline void launch_tiny(Ptr2 in, Ptr2 out, const LimbBatch& b, const NttTables& t,
                        cudaStream_t stream) {
  launch(ntt_tiny_kernel<INV>, b.count, t.n <= 64 ? 32 : t.n / 2, 0, stream, in, out, b,
         INV ? t.inv : t.fwd, t.mods, t.inv_last, t.n, t.logn);
}

}  // namespace nttk
}  // namespace fhert
