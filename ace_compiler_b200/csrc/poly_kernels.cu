// Element-wise, permutation, rescale, base-conversion and key inner-product
// kernels over limb-major RNS polynomials.  Kernels take a LimbBatch (or a
// compact group descriptor) so that one launch covers all limbs -- and, for a
// ciphertext, both polynomials -- of an operation; the x dimension of the grid
// walks the N coefficients of a limb, the y dimension the limbs.
#include <algorithm>

#include "ntt_kernels.cuh"
#include "runtime.h"

namespace fhert {

namespace {

constexpr int kThreads = 256;

inline dim3 grid_for(uint32_t n, int per_thread, int limbs) {
  uint32_t per_block = kThreads * per_thread;
  return dim3((n + per_block - 1) / per_block, limbs);
}

__device__ __forceinline__ const u64* sel_a(const Ptr2& p, const LimbRef& lr, uint32_t n) {
  return p.p[lr.sel & 1] + (size_t)lr.a * n;
}
__device__ __forceinline__ const u64* sel_b(const Ptr2& p, const LimbRef& lr, uint32_t n) {
  return p.p[(lr.sel >> 1) & 1] + (size_t)lr.b * n;
}
__device__ __forceinline__ u64* sel_d(const Ptr2& p, const LimbRef& lr, uint32_t n) {
  return p.p[(lr.sel >> 2) & 1] + (size_t)lr.dst * n;
}

// ---- element-wise (hal/src/hal.c:15-121, poly/src/rns_poly.c:852-1054) ------

// What bounds these kernels is bytes in flight: every thread issues the loads of
// four 16-byte words per operand before the first result.  With one 8-byte word at
// a time and integer products throughout, the 9 products and 8 sums of a
// convolution row at N = 65536 took 185 us, with two words 140, with four 131.  A
// limb has at least four coefficients, so whole words always fit.
constexpr int kWords = 4;  // 16-byte words per thread

inline dim3 grid_words(uint32_t n, int limbs) {
  const uint32_t per_block = kThreads * kWords * 2;
  return dim3((n + per_block - 1) / per_block, limbs);
}
struct WordLoop {  // the words of this thread
  uint32_t at[kWords];
  bool     in[kWords];
  __device__ __forceinline__ explicit WordLoop(uint32_t n) {
#pragma unroll
    for (int k = 0; k < kWords; k++) {
      at[k] = (blockIdx.x * kWords + k) * kThreads + threadIdx.x;
      in[k] = at[k] < n / 2;
    }
  }
  __device__ __forceinline__ void load(ulonglong2 (&v)[kWords], const u64* p) const {
#pragma unroll
    for (int k = 0; k < kWords; k++)
      v[k] = in[k] ? reinterpret_cast<const ulonglong2*>(p)[at[k]] : make_ulonglong2(0, 0);
  }
};

template <int OP>
__global__ void __launch_bounds__(kThreads)
ew_kernel(Ptr2 res, Ptr2 a, Ptr2 b, u64 scalar, const __grid_constant__ LimbBatch batch,
          const DevModulus* __restrict__ mods, uint32_t n) {
  constexpr bool   two  = OP == EW_ADD || OP == EW_SUB || OP == EW_MUL || OP == EW_MULADD;
  constexpr bool   accu = OP == EW_MULADD || OP == EW_MULADD_SCALAR;
  const LimbRef    lr = batch.limb[blockIdx.y];
  const DevModulus m  = mods[lr.prime];
  u64*             pr = sel_d(res, lr, n);
  u64              sc = 0;
  if (!two) {
    // scalars arrive as signed 64-bit values; bring into [0, q)
    int64_t s = (int64_t)scalar % (int64_t)m.q;
    sc        = s < 0 ? (u64)(s + (int64_t)m.q) : (u64)s;
  }
  const WordLoop words(n);
  ulonglong2     x[kWords], y[kWords], r[kWords];
  words.load(x, sel_a(a, lr, n));
  if (two) words.load(y, sel_b(b, lr, n));
  if (accu) words.load(r, pr);
  const nttk::Product mul(m);
  auto one = [&](u64 x, u64 y, u64 r) {
    if (!two) y = sc;
    if (OP == EW_ADD || OP == EW_ADD_SCALAR) return add_mod(x, y, m.q);
    if (OP == EW_SUB) return sub_mod(x, y, m.q);
    const u64 p = mul(x, y);
    return accu ? add_mod(r, p, m.q) : p;
  };
#pragma unroll
  for (int k = 0; k < kWords; k++)
    if (words.in[k])
      reinterpret_cast<ulonglong2*>(pr)[words.at[k]] =
          make_ulonglong2(one(x[k].x, y[k].x, r[k].x), one(x[k].y, y[k].y, r[k].y));
}

// one reduced scalar per limb of the batch, passed by value
// (rns_poly.c Scalars_integer_add_poly / Scalars_integer_multiply_poly)
struct ScalarList {
  u64 v[kMaxLimbs];
};

template <bool MUL>
__global__ void __launch_bounds__(kThreads)
ew_scalars_kernel(Ptr2 res, Ptr2 a, const __grid_constant__ ScalarList sc,
                  const __grid_constant__ LimbBatch batch, const DevModulus* __restrict__ mods,
                  uint32_t n) {
  const LimbRef    lr = batch.limb[blockIdx.y];
  const DevModulus m  = mods[lr.prime];
  const u64        s  = sc.v[blockIdx.y];
  u64*             pr = sel_d(res, lr, n);
  const WordLoop   words(n);
  ulonglong2       x[kWords];
  words.load(x, sel_a(a, lr, n));
  const nttk::Product mul(m);
  auto one = [&](u64 v) { return MUL ? mul(v, s) : add_mod(v, s, m.q); };
#pragma unroll
  for (int k = 0; k < kWords; k++)
    if (words.in[k])
      reinterpret_cast<ulonglong2*>(pr)[words.at[k]] = make_ulonglong2(one(x[k].x), one(x[k].y));
}

// ---- automorphism in NTT form: a pure gather (hal.c:123-138) ----------------

__global__ void __launch_bounds__(kThreads)
automorphism_kernel(Ptr2 res, Ptr2 val, const uint32_t* __restrict__ table, LimbBatch batch,
                    uint32_t n) {
  const LimbRef lr = batch.limb[blockIdx.y];
  const u64*    pv = sel_a(val, lr, n);
  u64*          pr = sel_d(res, lr, n);
  for (uint32_t i = blockIdx.x * kThreads + threadIdx.x; i < n; i += gridDim.x * kThreads)
    pr[i] = pv[__ldg(table + i)];
}

__global__ void __launch_bounds__(kThreads)
mul_const_kernel(Ptr2 res, Ptr2 val, const Twiddle* __restrict__ consts, LimbBatch batch,
                 const DevModulus* __restrict__ mods, uint32_t n) {
  const LimbRef lr = batch.limb[blockIdx.y];
  const u64     q  = mods[lr.prime].q;
  const Twiddle c  = consts[lr.prime];
  const u64*    pv = sel_a(val, lr, n);
  u64*          pr = sel_d(res, lr, n);
  for (uint32_t i = blockIdx.x * kThreads + threadIdx.x; i < n; i += gridDim.x * kThreads)
    pr[i] = mul_shoup(pv[i], c.w, c.wp, q);
}

// ---- tensor product (ckks/src/evaluator.c:137-173) ---------------------------
// limb index = prime index = blockIdx.y; the middle term is summed before its one
// reduction.  Seven words move per coefficient; two coefficients per thread and
// double-precision products where the prime allows.

__global__ void __launch_bounds__(kThreads)
tensor_kernel(u64* d0, u64* d1, u64* d2, const u64* a0, const u64* a1, const u64* b0, const u64* b1,
              const DevModulus* __restrict__ mods, uint32_t n, int first_prime) {
  const DevModulus m   = mods[first_prime + blockIdx.y];
  const size_t     off = (size_t)blockIdx.y * (n / 2);
  const uint32_t   i   = blockIdx.x * kThreads + threadIdx.x;
  if (i >= n / 2) return;
  typedef ulonglong2 w2;
  const w2 x0 = reinterpret_cast<const w2*>(a0)[off + i], x1 = reinterpret_cast<const w2*>(a1)[off + i];
  const w2 y0 = reinterpret_cast<const w2*>(b0)[off + i], y1 = reinterpret_cast<const w2*>(b1)[off + i];
  w2 r0, r1, r2;
  if (m.kind == kNttFloat) {
    const nttk::ArithFp f(m);
    auto                one = [&](u64 p0, u64 p1, u64 q0, u64 q1, u64& o0, u64& o1, u64& o2) {
      const double u0 = f.load(p0), u1 = f.load(p1), v0 = f.load(q0), v1 = f.load(q1);
      o0 = f.word(f.mul(u0, v0));
      o2 = f.word(f.mul(u1, v1));
      o1 = f.canon(__dadd_rn(f.mul(u0, v1), f.mul(u1, v0)));
    };
    one(x0.x, x1.x, y0.x, y1.x, r0.x, r1.x, r2.x);
    one(x0.y, x1.y, y0.y, y1.y, r0.y, r1.y, r2.y);
  } else {
    auto one = [&](u64 p0, u64 p1, u64 q0, u64 q1, u64& o0, u64& o1, u64& o2) {
      o0 = mul_mod(p0, q0, m);
      o2 = mul_mod(p1, q1, m);
      u64 hi = 0, lo = 0;
      mac_128(hi, lo, p0, q1);
      mac_128(hi, lo, p1, q0);
      o1 = reduce_128(hi, lo, m);
    };
    one(x0.x, x1.x, y0.x, y1.x, r0.x, r1.x, r2.x);
    one(x0.y, x1.y, y0.y, y1.y, r0.y, r1.y, r2.y);
  }
  reinterpret_cast<w2*>(d0)[off + i] = r0;
  reinterpret_cast<w2*>(d1)[off + i] = r1;
  reinterpret_cast<w2*>(d2)[off + i] = r2;
}

// ---- rescale (rns_poly.c:351-383) -------------------------------------------

__global__ void __launch_bounds__(kThreads)
rescale_lift_kernel(Ptr2 tmp, Ptr2 last, u64 q_last, const Twiddle* __restrict__ neg_row,
                    const u64* __restrict__ mod_row, LimbBatch batch,
                    const DevModulus* __restrict__ mods, uint32_t n) {
  const LimbRef    lr = batch.limb[blockIdx.y];
  const DevModulus m  = mods[lr.prime];
  const Twiddle    w  = neg_row[lr.prime];
  const u64        om = mod_row[lr.prime];
  const u64*       pl = sel_b(last, lr, n);
  u64*             pt = sel_d(tmp, lr, n);
  for (uint32_t i = blockIdx.x * kThreads + threadIdx.x; i < n; i += gridDim.x * kThreads) {
    u64 s = switch_modulus(pl[i], q_last, m, om);
    pt[i] = mul_shoup(s, w.w, w.wp, m.q);
  }
}

__global__ void __launch_bounds__(kThreads)
rescale_combine_kernel(Ptr2 res, Ptr2 poly, Ptr2 tmp, const Twiddle* __restrict__ inv_row,
                       LimbBatch batch, const DevModulus* __restrict__ mods, uint32_t n) {
  const LimbRef lr = batch.limb[blockIdx.y];
  const u64     q  = mods[lr.prime].q;
  const Twiddle w  = inv_row[lr.prime];
  const u64*    pp = sel_a(poly, lr, n);
  const u64*    pt = sel_b(tmp, lr, n);
  u64*          pr = sel_d(res, lr, n);
  for (uint32_t i = blockIdx.x * kThreads + threadIdx.x; i < n; i += gridDim.x * kThreads)
    pr[i] = add_mod(mul_shoup(pp[i], w.w, w.wp, q), pt[i], q);
}

// ---- ModDown tail (rns_poly.c:293-304), optionally adding a polynomial -------

__global__ void __launch_bounds__(kThreads)
moddown_combine_kernel(ModDownTail a, const Twiddle* __restrict__ p_inv,
                       const DevModulus* __restrict__ mods, uint32_t n) {
  const int     g   = blockIdx.z;
  if ((a.skip_mask >> blockIdx.y) & 1) return;
  const u64     q   = mods[blockIdx.y].q;
  const Twiddle w   = p_inv[blockIdx.y];
  const size_t  off = (size_t)blockIdx.y * n;
  const u64*    px  = a.x[g] + off;
  const u64*    pt  = a.t[g] + off;
  const u64*    pa  = a.add[g] ? a.add[g] + off : nullptr;
  u64*          pr  = a.res[g] + off;
  for (uint32_t i = blockIdx.x * kThreads + threadIdx.x; i < n; i += gridDim.x * kThreads) {
    u64 r = mul_shoup(sub_mod(px[i], pt[i], q), w.w, w.wp, q);
    if (pa) r = add_mod(r, pa[i], q);
    pr[i] = r;
  }
}

// ---- fused ModDown + Rescale tail, coefficient form (rns_poly.c:556-596) -----

// Sub_mul_const_mod of the CPU runtime (modular.h:266-276) on operands where
// val2 may exceed the modulus: the signed difference gets the modulus added
// once when negative and may stay negative; the Shoup product then runs on its
// two's-complement image exactly as the 128-bit host arithmetic does.
__device__ __forceinline__ u64 sub_mul_const_exact(u64 v1, u64 v2, u64 w, u64 wp, u64 q) {
  long long s = (long long)v1 - (long long)v2;
  if (s < 0) s += (long long)q;
  u64 lo = (u64)s;
  u64 qt = __umul64hi(lo, wp) - (s < 0 ? wp : 0);  // ((2^128 + s) * wp >> 64) mod 2^64
  u64 y  = lo * w - qt * q;
  return y >= q ? y - q : y;
}

__global__ void __launch_bounds__(kThreads)
moddown_rescale_kernel(u64* __restrict__ res, const u64* __restrict__ x,
                       const u64* __restrict__ t, int last, const Twiddle* __restrict__ p_inv,
                       const Twiddle* __restrict__ ql_inv_row,
                       const DevModulus* __restrict__ mods, uint32_t n) {
  const int     i    = blockIdx.y;  // output limb, i < last
  const u64     q    = mods[i].q, ql = mods[last].q;
  const Twiddle pi   = p_inv[i], pl = p_inv[last], wi = ql_inv_row[i];
  const u64*    xi   = x + (size_t)i * n;
  const u64*    ti   = t + (size_t)i * n;
  const u64*    xl   = x + (size_t)last * n;
  const u64*    tl   = t + (size_t)last * n;
  u64*          ri   = res + (size_t)i * n;
  for (uint32_t k = blockIdx.x * kThreads + threadIdx.x; k < n; k += gridDim.x * kThreads) {
    u64 last_new = mul_shoup(sub_mod(xl[k], tl[k], ql), pl.w, pl.wp, ql);
    u64 nv       = mul_shoup(sub_mod(xi[k], ti[k], q), pi.w, pi.wp, q);
    ri[k]        = sub_mul_const_exact(nv, last_new, wi.w, wi.wp, q);
  }
}

// Rescale of a polynomial in coefficient form (rns_poly.c:381-399): the dropped
// limb is reduced as it stands (no centring, unlike the NTT-form branch),
// res_i = (x_i - (x_last mod q_i)) * q_last^-1 mod q_i.  blockIdx.y runs over
// the limbs of `polys` polynomials of `last` output limbs each.
__global__ void __launch_bounds__(kThreads)
rescale_coeff_kernel(Ptr2 res, Ptr2 x, int last, const Twiddle* __restrict__ ql_inv_row,
                     const DevModulus* __restrict__ mods, uint32_t n) {
  const int        g  = blockIdx.y / last, i = blockIdx.y % last;
  const DevModulus md = mods[i];
  const Twiddle    wi = ql_inv_row[i];
  const u64*       xi = (g ? x.p[1] : x.p[0]) + (size_t)i * n;
  const u64*       xl = (g ? x.p[1] : x.p[0]) + (size_t)last * n;
  u64*             ri = (g ? res.p[1] : res.p[0]) + (size_t)i * n;
  for (uint32_t k = blockIdx.x * kThreads + threadIdx.x; k < n; k += gridDim.x * kThreads)
    ri[k] = mul_shoup(sub_mod(xi[k], reduce_128(0, xl[k], md), md.q), wi.w, wi.wp, md.q);
}

// ---- mod-raise (rns_poly.c:1101-1125) ----------------------------------------

__global__ void __launch_bounds__(kThreads)
mod_raise_kernel(u64* __restrict__ res, const u64* __restrict__ src, u64 q0,
                 LimbBatch batch, const DevModulus* __restrict__ mods, uint32_t n) {
  const LimbRef    lr = batch.limb[blockIdx.y];
  const DevModulus m  = mods[lr.prime];
  const u64        om = q0 % m.q;
  u64*             pr = res + (size_t)lr.dst * n;
  for (uint32_t i = blockIdx.x * kThreads + threadIdx.x; i < n; i += gridDim.x * kThreads)
    pr[i] = lr.prime == 0 ? src[i] : switch_modulus(src[i], q0, m, om);
}

inline void after_launch(Context* c, KernelId id, int limbs) {
  prof_after(id, limbs);
  c->launches++;
  CUDA_CHECK(cudaGetLastError());
}

}  // namespace

void launch_elementwise(EwOp op, Ptr2 res, Ptr2 a, Ptr2 b, int64_t scalar,
                        const LimbBatch& batch) {
  if (batch.count == 0) return;
  Context* c = ctx();
  DagScope dag(DAG_ELEMENTWISE);
  {
    const bool two  = op == EW_ADD || op == EW_SUB || op == EW_MUL || op == EW_MULADD;
    const bool accu = op == EW_MULADD || op == EW_MULADD_SCALAR;
    dag.batch(batch, c->N, &res, &a, two ? &b : nullptr, accu);
  }
  dag.commit();
  prof_before(KID_ELEMENTWISE);
  dim3 g = grid_words(c->N, batch.count);
#define EW_CASE(OP)                                                                        \
  case OP:                                                                                 \
    launch(ew_kernel<OP>, g, kThreads, 0, c->stream, res, a, b, (u64)scalar, batch, c->d_mod, c->N);                                    \
    break;
  switch (op) {
    EW_CASE(EW_ADD)
    EW_CASE(EW_SUB)
    EW_CASE(EW_MUL)
    EW_CASE(EW_MULADD)
    EW_CASE(EW_ADD_SCALAR)
    EW_CASE(EW_MUL_SCALAR)
    EW_CASE(EW_MULADD_SCALAR)
  }
#undef EW_CASE
  after_launch(c, KID_ELEMENTWISE, batch.count);
}

void launch_scalars(bool mul, Ptr2 res, Ptr2 a, const u64* per_limb, const LimbBatch& batch) {
  if (batch.count == 0) return;
  Context* c = ctx();
  ScalarList sc;
  for (int i = 0; i < batch.count; i++) sc.v[i] = per_limb[i];
  DagScope dag(DAG_PER_LIMB_CONST);
  dag.batch(batch, c->N, &res, &a, nullptr);
  dag.commit();
  prof_before(KID_ELEMENTWISE);
  dim3 g = grid_words(c->N, batch.count);
  if (mul) launch(ew_scalars_kernel<true>, g, kThreads, 0, c->stream,
                  res, a, sc, batch, c->d_mod, c->N);
  else launch(ew_scalars_kernel<false>, g, kThreads, 0, c->stream,
              res, a, sc, batch, c->d_mod, c->N);
  after_launch(c, KID_ELEMENTWISE, batch.count);
}

void launch_automorphism(Ptr2 res, Ptr2 val, const uint32_t* table, const LimbBatch& batch) {
  if (batch.count == 0) return;
  Context* c = ctx();
  DagScope dag(DAG_AUTOMORPHISM);
  dag.batch(batch, c->N, &res, &val, nullptr);
  dag.commit();
  prof_before(KID_AUTOMORPHISM);
  launch(automorphism_kernel, grid_for(c->N, 2, batch.count), kThreads, 0, c->stream,
         res, val, table, batch, c->N);
  after_launch(c, KID_AUTOMORPHISM, batch.count);
}

void launch_mul_const(Ptr2 res, Ptr2 val, const Twiddle* consts, const LimbBatch& batch) {
  if (batch.count == 0) return;
  Context* c = ctx();
  DagScope dag(DAG_PER_LIMB_CONST);
  dag.batch(batch, c->N, &res, &val, nullptr);
  dag.commit();
  prof_before(KID_MUL_CONST);
  launch(mul_const_kernel, grid_for(c->N, 2, batch.count), kThreads, 0, c->stream,
         res, val, consts, batch, c->d_mod, c->N);
  after_launch(c, KID_MUL_CONST, batch.count);
}

void launch_tensor_range(int64_t* d0, int64_t* d1, int64_t* d2, const int64_t* a0,
                         const int64_t* a1, const int64_t* b0, const int64_t* b1, int first_prime,
                         int count) {
  if (count == 0) return;
  Context* c = ctx();
  DagScope dag(DAG_TENSOR);
  if (dag.live) {
    const size_t bytes = (size_t)count * c->N * sizeof(int64_t);
    for (const int64_t* r : {a0, a1, b0, b1}) dag.set.read(r, bytes);
    for (int64_t* w : {d0, d1, d2}) dag.set.write(w, bytes);
  }
  dag.commit();
  prof_before(KID_TENSOR);
  launch(tensor_kernel, grid_for(c->N, 2, count), kThreads, 0, c->stream,
         (u64*)d0, (u64*)d1, (u64*)d2, (const u64*)a0, (const u64*)a1, (const u64*)b0,
         (const u64*)b1, c->d_mod, c->N, first_prime);
  after_launch(c, KID_TENSOR, count);
}

void launch_tensor(int64_t* d0, int64_t* d1, int64_t* d2, const int64_t* a0,
                   const int64_t* a1, const int64_t* b0, const int64_t* b1, int level) {
  launch_tensor_range(d0, d1, d2, a0, a1, b0, b1, 0, level);
}

void launch_rescale_lift(Ptr2 tmp, Ptr2 last, int l, const LimbBatch& batch) {
  if (batch.count == 0) return;
  Context* c = ctx();
  prof_before(KID_RESCALE_LIFT);
  launch(rescale_lift_kernel, grid_for(c->N, 2, batch.count), kThreads, 0, c->stream,
         tmp, last, c->primes[l], c->d_ql_neg + (size_t)l * c->L, c->d_ql_mod + (size_t)l * c->L,
         batch, c->d_mod, c->N);
  after_launch(c, KID_RESCALE_LIFT, batch.count);
}

void launch_rescale_combine(Ptr2 res, Ptr2 poly, Ptr2 tmp, int l, const LimbBatch& batch) {
  if (batch.count == 0) return;
  Context* c = ctx();
  prof_before(KID_RESCALE_COMBINE);
  launch(rescale_combine_kernel, grid_for(c->N, 2, batch.count), kThreads, 0, c->stream,
         res, poly, tmp, c->d_ql_inv + (size_t)l * c->L, batch, c->d_mod, c->N);
  after_launch(c, KID_RESCALE_COMBINE, batch.count);
}

void launch_moddown_combine(const ModDownTail& args) {
  if (args.level == 0 || args.polys == 0) return;
  Context* c = ctx();
  prof_before(KID_MODDOWN_COMBINE);
  dim3 g = grid_for(c->N, 2, args.level);
  g.z    = args.polys;
  launch(moddown_combine_kernel, g, kThreads, 0, c->stream, args, c->d_p_inv, c->d_mod, c->N);
  after_launch(c, KID_MODDOWN_COMBINE, args.level * args.polys);
}

void launch_moddown_rescale(int64_t* res, const int64_t* x, const int64_t* t, int level) {
  if (level < 2) return;
  Context* c    = ctx();
  const int last = level - 1;
  prof_before(KID_MODDOWN_COMBINE);
  launch(moddown_rescale_kernel, grid_for(c->N, 2, last), kThreads, 0, c->stream,
         (u64*)res, (const u64*)x, (const u64*)t, last, c->d_p_inv,
         c->d_ql_inv + (size_t)last * c->L, c->d_mod, c->N);
  after_launch(c, KID_MODDOWN_COMBINE, last);
}

void launch_rescale_coeff(Ptr2 res, Ptr2 x, int polys, int level) {
  if (level < 2) return;
  Context*  c    = ctx();
  const int last = level - 1;
  prof_before(KID_RESCALE_COMBINE);
  launch(rescale_coeff_kernel, grid_for(c->N, 2, polys * last), kThreads, 0, c->stream,
         res, x, last, c->d_ql_inv + (size_t)last * c->L, c->d_mod, c->N);
  after_launch(c, KID_RESCALE_COMBINE, polys * last);
}

void launch_mod_raise(int64_t* res, const int64_t* src, const LimbBatch& batch) {
  if (batch.count == 0) return;
  Context* c = ctx();
  DagScope dag(DAG_PER_LIMB_CONST);
  if (dag.live) {
    const size_t w = (size_t)c->N * sizeof(int64_t);
    dag.set.read(src, w);
    for (int i = 0; i < batch.count; i++) dag.set.write(res + (size_t)batch.limb[i].dst * c->N, w);
  }
  dag.commit();
  prof_before(KID_MOD_RAISE);
  launch(mod_raise_kernel, grid_for(c->N, 2, batch.count), kThreads, 0, c->stream,
         (u64*)res, (const u64*)src, c->primes[0], batch, c->d_mod, c->N);
  after_launch(c, KID_MOD_RAISE, batch.count);
}

}  // namespace fhert
