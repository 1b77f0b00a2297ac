// Approximate base conversion of ModUp and ModDown on the tensor cores
// (rns_poly.c:218-242, rns_poly_impl.c:287-339 of the CPU runtime):
//   y_i      = in_i * inv_i mod p_i            (canonical residues, up to 16 limbs;
//              no inv: the inverse transform before has multiplied already)
//   out_m    = (sum_i y_i * mat_{i,m}) mod q_m  for up to 60 output primes m.
//
// Written with the bytes of y_i the sum is
//   sum_{i,b} byte_b(y_i) * (2^{8b} mat_{i,m} mod q_m),
// and with the bytes of the constants in parentheses it becomes one product of
// unsigned bytes per coefficient, output and byte plane s of the result,
//   D_s = sum_{i,b} byte_b(y_i) * byte_s(2^{8b} mat_{i,m} mod q_m)  < 2^23,
//   out_m = (sum_s 2^{8s} D_s) mod q_m,
// exact in 32-bit accumulators.  That is a matrix product of (coefficients) x
// (8 bytes per input limb) x (8 planes per output): tcgen05.mma kind::i8 with
// 128 coefficients as rows, the words y_i themselves as the K bytes, and the 8
// planes of an output in 8 neighbouring columns, so that a thread reads all
// planes of its coefficient from tensor memory and finishes with some 25
// integer instructions instead of 4 multiply-adds per input and output plus a
// 128-bit reduction (about 130 at 12 inputs, bound by the integer multiplier:
// 63 % of the launch).
//
// A CTA takes 256 coefficients (two row tiles) and all outputs of one group, 8
// outputs (64 columns) at a time: 128 columns of tensor memory, four CTAs per SM,
// so that one CTA's products run under the others' reductions.  What bounds it
// is the issue rate of those reductions (59 instructions per output word, 57 % of
// the issue slots; ModUp and ModDown of a rotation at 36 limbs of N = 65536 took
// 164 us with multiply-adds, 46 here).  Four outputs per product with two products
// in turn (29 us), and the outputs split over two to four CTAs (30 to 32), lost.
#include <algorithm>
#include <vector>

#include "ntt_kernels.cuh"
#include "runtime.h"

namespace fhert {

namespace {

using nttk::csub;

constexpr int kThreads = 256;
constexpr int kRows    = 128;  // coefficients per matrix product
constexpr int kOuts    = 8;    // outputs per product: 64 columns
constexpr int kColumns = 128;  // tensor memory of a CTA: two row tiles
// 2 us a poll: a wait that lasts longer than any product by orders of magnitude
constexpr uint32_t kMaxPolls = 1u << 15;

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  for (uint32_t k = 0; k < kMaxPolls; k++) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, 2000;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// K-major operand without swizzle: 8 x 16-byte core matrices of 128 bytes, `lead`
// bytes apart along K, `stride` bytes apart along the rows
__device__ __forceinline__ u64 operand_desc(uint32_t addr, uint32_t lead, uint32_t stride) {
  return (u64)((addr >> 4) & 0x3fff) | ((u64)((lead >> 4) & 0x3fff) << 16) |
         ((u64)((stride >> 4) & 0x3fff) << 32) | (1ull << 46);
}
// unsigned bytes, 32-bit sums, 128 rows, `columns` columns
__device__ __forceinline__ uint32_t product_desc(uint32_t columns) {
  return (2u << 4) | ((columns >> 3) << 17) | ((uint32_t)(kRows >> 4) << 24);
}
__device__ __forceinline__ void product(uint32_t d, u64 a, u64 b, uint32_t desc, uint32_t add) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
      "l"(a), "l"(b), "r"(desc), "r"(add)
      : "memory");
}
// 32 columns of this warp's 32 lanes
__device__ __forceinline__ void tmem_load32(uint32_t (&v)[32], uint32_t addr) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
        "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
        "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]),
        "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]),
        "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(addr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

struct OutConst {  // one output of the group
  u64      q, nq;   // modulus, 2^64 - q
  u64*     dst;     // its limb; nullptr = computed elsewhere (or padding)
  uint32_t mu, shift;
};

// (sum_s 2^{8s} D_s) mod q.  V < 2^{8S+15} for S planes; the quotient is estimated
// from the 32 bits of V above shift = 8S - 16 and mu = floor(2^{32+shift} / q): it
// is at most 1.51 too small, one subtraction is left.  WIDE: seven or eight planes.
template <bool WIDE>
__device__ __forceinline__ u64 reduce_planes(const uint32_t* d, const OutConst& c) {
  const uint32_t u0 = d[0] + (d[1] << 8), u1 = d[2] + (d[3] << 8), u2 = d[4] + (d[5] << 8);
  u64            a;
  asm("mad.wide.u32 %0, %1, 65536, %2;" : "=l"(a) : "r"(u1), "l"((u64)u0));
  const uint32_t w0 = (uint32_t)a;
  uint32_t       w1, top;
  if (WIDE) {
    const uint32_t u3 = d[6] + (d[7] << 8);
    u64            b;
    asm("mad.wide.u32 %0, %1, 65536, %2;" : "=l"(b) : "r"(u3), "l"((u64)u2));
    const u64 mid = (a >> 32) + (uint32_t)b;
    w1            = (uint32_t)mid;
    top           = __funnelshift_rc(w1, (uint32_t)(b >> 32) + (uint32_t)(mid >> 32), c.shift - 32);
  } else {
    w1  = (uint32_t)(a >> 32) + u2;
    top = __funnelshift_rc(w0, w1, c.shift);
  }
  const uint32_t k = __umulhi(top, c.mu);
  u64            r;
  asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(r) : "r"(k), "r"((uint32_t)c.nq), "l"(((u64)w1 << 32) | w0));
  uint32_t rh = (uint32_t)(r >> 32);
  asm("mad.lo.u32 %0, %1, %2, %0;" : "+r"(rh) : "r"(k), "r"((uint32_t)(c.nq >> 32)));
  r                 = ((u64)rh << 32) | (uint32_t)r;
  const long long t = (long long)(r - c.q);  // r < 2q < 2^63
  return t < 0 ? r : (u64)t;
}

template <bool WIDE>
__device__ __forceinline__ void finish4(const uint32_t (&d)[32], const OutConst* c, uint32_t coeff,
                                        bool live) {
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const u64 r = reduce_planes<WIDE>(d + 8 * j, c[j]);
    if (c[j].dst != nullptr && live) c[j].dst[coeff] = r;
  }
}

// NIN: input limbs rounded up to a multiple of four (32 K bytes per product step)
template <int NIN>
__global__ void __launch_bounds__(kThreads, 4)
base_conv_kernel(const __grid_constant__ ConvArgs args, int num_q, const DevModulus* __restrict__ mods,
                 uint32_t n, uint32_t* error) {
  constexpr int kBytes = NIN * 8;        // K bytes per row
  constexpr int kGroup = kBytes * 8;     // bytes of 8 rows: one output's planes, 8 coefficients
  extern __shared__ __align__(128) unsigned char dyn[];
  __shared__ OutConst  outs[kMaxOuts + 4];
  __shared__ __align__(8) u64 bars[2];
  __shared__ uint32_t  tmem_slot, failed;

  const ConvGroup& g         = args.g[blockIdx.y];
  const int        out_count = args.out_total - g.skip_len;
  unsigned char*   a_mem     = dyn;                              // [2][128 rows]
  unsigned char*   b_mem     = dyn + 2 * kRows * kBytes;         // [out_count (+1)] planes
  const uint32_t   load_bar = smem_addr(&bars[0]), mma_bar = smem_addr(&bars[1]);
  const int        warp = threadIdx.x >> 5, row = threadIdx.x & (kRows - 1), tile = threadIdx.x >> 7;

  if (threadIdx.x == 0) {
    failed = 0;
    mbar_init(load_bar, 1);
    mbar_init(mma_bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    const uint32_t bytes = (uint32_t)(out_count * kGroup);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(load_bar), "r"(bytes)
                 : "memory");
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_addr(b_mem)),
        "l"(g.planes), "r"(bytes), "r"(load_bar)
        : "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_addr(&tmem_slot)),
                 "r"((uint32_t)kColumns)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  for (int o = threadIdx.x; o < ((out_count + 3) & ~3); o += kThreads) {
    const bool real = o < out_count;  // padding looks like the last output
    const int  at   = real ? o : out_count - 1;
    const int  m    = at < g.skip_start ? at : at + g.skip_len;
    const bool is_q = m < args.level;
    const DevModulus& md = mods[is_q ? m : num_q + (m - args.level)];
    const int  limb = is_q ? m : args.p_limb + (m - args.level);
    OutConst   c;
    c.q     = md.q;
    c.nq    = 0 - md.q;
    c.mu    = md.conv_mu;
    c.shift = md.conv_shift;
    c.dst   = !real || (m < 64 && ((args.skip_mask >> m) & 1)) ? nullptr : g.out + (size_t)limb * n;
    outs[o] = c;
  }

  // y_i of this thread's coefficient, as the row's K bytes
  const uint32_t coeff = blockIdx.x * kThreads + threadIdx.x;
  const bool     live  = coeff < n;
  u64            y[NIN];
#pragma unroll
  for (int i = 0; i < NIN; i++)
    y[i] = live && i < g.count ? g.in[(size_t)(g.first_limb + i) * n + coeff] : 0;
  if (g.inv != nullptr) {
#pragma unroll
    for (int i = 0; i < NIN; i++) {
      if (i >= g.count) break;
      const nttk::Mod m = nttk::make_mod(mods[g.first_prime + i].q);
      y[i] = nttk::canon_4q(nttk::shoup4(y[i], nttk::ld_tw(g.inv + i), m), m);
    }
  }
  {
    unsigned char* at = a_mem + tile * (kRows * kBytes) + (row >> 3) * kGroup + (row & 7) * 16;
#pragma unroll
    for (int i = 0; i < NIN; i += 2)
      *reinterpret_cast<ulonglong2*>(at + (i >> 1) * 128) = make_ulonglong2(y[i], y[i + 1]);
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot;

  for (int o0 = 0, phase = 0; o0 < out_count; o0 += kOuts, phase ^= 1) {
    const int here = min(kOuts, out_count - o0);
    if (threadIdx.x == 0) {
      if (o0 == 0 && !mbar_wait(load_bar, 0)) failed = 1;
      const uint32_t columns = (uint32_t)((here + 1) & ~1) * 8, desc = product_desc(columns);
#pragma unroll
      for (int t = 0; t < 2; t++)
#pragma unroll
        for (int k = 0; k < kBytes / 32; k++)
          product(tmem + t * (kColumns / 2),
                  operand_desc(smem_addr(a_mem) + t * (kRows * kBytes) + k * 256, 128, kGroup),
                  operand_desc(smem_addr(b_mem) + o0 * kGroup + k * 256, 128, kGroup), desc, k > 0);
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                       mma_bar)
                   : "memory");
    }
    if (!mbar_wait(mma_bar, (uint32_t)phase)) failed = 1;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t at = tmem + tile * (kColumns / 2) + ((uint32_t)(warp & 3) << 21);
    for (int o = 0; o < here; o += 4) {
      uint32_t d[32];
      tmem_load32(d, at + o * 8);
      const OutConst* c = outs + o0 + o;
      // outputs of one group are alike but for a prime or two
      const uint32_t widest = max(max(c[0].shift, c[1].shift), max(c[2].shift, c[3].shift));
      if (widest <= 32) {
        finish4<false>(d, c, coeff, live);
      } else if (min(min(c[0].shift, c[1].shift), min(c[2].shift, c[3].shift)) > 32) {
        finish4<true>(d, c, coeff, live);
      } else {
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const u64 r = c[j].shift > 32 ? reduce_planes<true>(d + 8 * j, c[j]) : reduce_planes<false>(d + 8 * j, c[j]);
          if (c[j].dst != nullptr && live) c[j].dst[coeff] = r;
        }
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();  // the next product overwrites these columns
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (failed) break;
  }
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"((uint32_t)kColumns));
  if (threadIdx.x == 0 && failed) atomicExch(error, 1u);
}

template <int NIN>
void dispatch(Context* c, const ConvArgs& args, int max_out) {
  // one output more than there are: an odd count is rounded up to 16 columns
  const size_t smem = (size_t)2 * kRows * NIN * 8 + (size_t)(max_out + 1) * NIN * 64;
  static size_t allowed = 44 * 1024;  // without asking, 48 KiB less the static part
  if (smem > allowed) {
    CUDA_CHECK(cudaFuncSetAttribute(base_conv_kernel<NIN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)smem));
    allowed = smem;
  }
  launch(base_conv_kernel<NIN>, dim3((c->N + kThreads - 1) / kThreads, args.groups), kThreads, smem,
         c->stream, args, c->L, c->d_mod, c->N, c->d_error);
}

}  // namespace

std::vector<uint8_t> conv_planes(int inputs, int width, int outputs, const u64* mat, const u64* primes) {
  std::vector<uint8_t> planes((size_t)outputs * width * 64, 0);
  for (int o = 0; o < outputs; o++)
    for (int i = 0; i < inputs; i++) {
      u64 v = mat[(size_t)o * inputs + i];
      for (int b = 0; b < 8; b++) {
        // byte b of y_i is K byte 8i + b: core matrix (8i + b) / 16, column % 16
        const int kb = 8 * i + b;
        uint8_t*  at = &planes[(size_t)o * width * 64 + (size_t)(kb / 16) * 128 + kb % 16];
        for (int s = 0; s < 8; s++) at[s * 16] = (uint8_t)(v >> (8 * s));
        v = mulmod(v, 256, primes[o]);
      }
    }
  return planes;
}

void launch_base_conv(const ConvArgs& args) {
  Context* c = ctx();
  int max_in = 0, max_out = 0, total_out = 0;
  for (int g = 0; g < args.groups; g++) {
    max_in  = std::max(max_in, args.g[g].count);
    max_out = std::max(max_out, args.out_total - args.g[g].skip_len);
    total_out += args.out_total - args.g[g].skip_len;
  }
  if (max_out <= 0 || args.groups == 0) return;
  FHERT_ASSERT(max_in <= args.width && args.width <= kMaxDigit && max_out <= kMaxOuts,
               "base conversion from %d to %d limbs unsupported", max_in, max_out);
  DagScope dag(DAG_BASE_CONV);
  if (dag.live) {
    const size_t w = (size_t)c->N * sizeof(u64);
    for (int g = 0; g < args.groups; g++) {
      const ConvGroup& cg = args.g[g];
      dag.set.read(cg.in + (size_t)cg.first_limb * c->N, (size_t)cg.count * w);
      for (int m = 0; m < args.out_total; m++) {
        if (m >= cg.skip_start && m < cg.skip_start + cg.skip_len) continue;
        if (m < 64 && ((args.skip_mask >> m) & 1)) continue;
        int limb = m < args.level ? m : args.p_limb + (m - args.level);
        dag.set.write(cg.out + (size_t)limb * c->N, w);
      }
    }
  }
  dag.commit();
  prof_before(KID_BASE_CONV);
  if (args.width == 4) dispatch<4>(c, args, max_out);
  else if (args.width == 8) dispatch<8>(c, args, max_out);
  else if (args.width == 12) dispatch<12>(c, args, max_out);
  else dispatch<16>(c, args, max_out);
  c->launches++;
  prof_after(KID_BASE_CONV, total_out);
  CUDA_CHECK(cudaGetLastError());
}

}  // namespace fhert
