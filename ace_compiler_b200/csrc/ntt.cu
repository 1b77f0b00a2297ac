// Negacyclic NTT / inverse NTT over one or many RNS limbs: launch side.
// The kernels and the arithmetic are in ntt_kernels.cuh.
#include <algorithm>

#include "ntt_kernels.cuh"

namespace fhert {

namespace {

// The two-pass kernels want the limbs transformed in integers first (they take
// longest, the others fill up behind them); returns how many there are.
int integers_first(Context* c, LimbBatch& b) {
  auto* mid = std::stable_partition(b.limb, b.limb + b.count,
                                    [&](const LimbRef& r) { return !c->ntt_float[r.prime]; });
  return (int)(mid - b.limb);
}

template <bool INV>
void launch_dir(Ptr2 in, Ptr2 out, const LimbBatch& unsorted, const Twiddle* last) {
  Context*        c = ctx();
  LimbBatch       b = unsorted;
  nttk::NttTables t{c->d_fwd, c->d_inv, last ? last : c->d_inv_last, c->d_mod, c->N, (int)c->logN};
  if (t.logn <= nttk::kWholeMaxLog) {  // one launch
    DagScope dag(DAG_NTT);
    dag.batch(b, c->N, &out, &in, nullptr);
    dag.commit();
    prof_before(INV ? KID_INTT_SMALL : KID_NTT_SMALL);
    if (t.logn <= nttk::kTinyMaxLog) nttk::launch_tiny<INV>(in, out, b, t, c->stream);
    else nttk::launch_whole<INV>(in, out, b, t, c->stream);
    prof_after(INV ? KID_INTT_SMALL : KID_NTT_SMALL, b.count);
    c->launches++;
    CUDA_CHECK(cudaGetLastError());
    return;
  }
  const int n_int = integers_first(c, b);
  // the second pass works in place on `out`
  LimbBatch b2 = b;
  for (int i = 0; i < b2.count; i++) {
    b2.limb[i].a   = b2.limb[i].dst;
    b2.limb[i].sel = (uint8_t)((b2.limb[i].sel & 4) | ((b2.limb[i].sel >> 2) & 1));
  }
  // both passes under one description: the second works in place on what the first wrote
  DagScope dag(DAG_NTT);
  dag.batch(b, c->N, &out, &in, nullptr);
  dag.commit();
  if (!INV) {
    prof_before(KID_NTT_STRIDED);
    nttk::launch_strided<false>(in, out, b, n_int, t, c->stream);
    prof_after(KID_NTT_STRIDED, b.count);
    prof_before(KID_NTT_CONTIG);
    nttk::launch_contig<false>(out, out, b2, n_int, t, c->stream);
    prof_after(KID_NTT_CONTIG, b.count);
  } else {
    prof_before(KID_INTT_CONTIG);
    nttk::launch_contig<true>(in, out, b, n_int, t, c->stream);
    prof_after(KID_INTT_CONTIG, b.count);
    prof_before(KID_INTT_STRIDED);
    nttk::launch_strided<true>(out, out, b2, n_int, t, c->stream);
    prof_after(KID_INTT_STRIDED, b.count);
  }
  c->launches += 2;
  CUDA_CHECK(cudaGetLastError());
}

}  // namespace

bool ntt_can_fuse() { return (int)ctx_noflush()->logN > nttk::kTinyMaxLog; }

void launch_ntt_fused(Ptr2 in, int64_t* mid, Ptr2 out, const LimbBatch& b, const NttFuse& f) {
  if (b.count == 0) return;
  Context*        c = ctx();
  nttk::NttTables t{c->d_fwd, c->d_inv, c->d_inv_last, c->d_mod, c->N, (int)c->logN};
  FHERT_ASSERT(t.logn > nttk::kTinyMaxLog, "ring degree too small for a fused transform");
  nttk::NttPro pro;
  pro.kind   = f.pro_kind;
  pro.mul    = f.pro_mul;
  pro.mod    = f.pro_mod;
  pro.q_last = f.q_last;
  pro.last_x    = f.last_x;
  pro.last_conv = f.last_conv;
  pro.twice     = f.twice;
  nttk::NttEpi epi;
  epi.kind = f.epi_kind;
  epi.mul  = f.epi_mul;
  epi.aux  = f.aux;
  epi.add  = f.add;
  epi.perm = f.perm;
  // strided pass: in[a] -> mid[k] (mid[a] with prologue 3); contiguous pass: from there
  // to out[dst] with the epilogue
  LimbBatch b1 = b, b2 = b;
  for (int i = 0; i < b.count; i++) {
    const uint16_t mid_limb = (uint16_t)(f.pro_kind == 3 ? b.limb[i].a : i);
    b1.limb[i].dst = mid_limb;
    b1.limb[i].sel = (uint8_t)(f.multi ? 0 : b.limb[i].sel & 1);
    b2.limb[i].a   = mid_limb;
    b2.limb[i].sel = (uint8_t)(f.multi ? b.limb[i].sel : b.limb[i].sel & 6);
  }
  const int n_int = integers_first(c, b1);
  integers_first(c, b2);
  DagScope dag(DAG_NTT_FUSED);
  if (dag.live) {
    const size_t w = (size_t)c->N * sizeof(u64);
    for (int i = 0; i < b.count; i++) dag.set.write(mid + (size_t)b1.limb[i].dst * c->N, w);
    for (int g = 0; g < 2 && f.pro_kind == 3; g++) {
      dag.set.read(f.last_x.p[g], w);
      dag.set.read(f.last_conv.p[g], w);
    }
    if (f.multi == nullptr) dag.batch(b, c->N, &out, &in, nullptr);
    for (int i = 0; i < b.count; i++) {
      const LimbRef& lr = b.limb[i];
      const size_t   at = (size_t)lr.b * c->N;
      if (f.multi != nullptr) {
        const size_t to = (size_t)lr.dst * c->N;
        dag.set.read(in.p[0] + (size_t)lr.a * c->N, w);
        dag.set.read(f.aux.p[0] + at, w);
        if (f.multi->add[lr.sel] != nullptr) dag.set.read(f.multi->add[lr.sel] + to, w);
        dag.set.write(f.multi->out[lr.sel] + to, w);
      } else if (f.epi_kind != 0) {
        dag.set.read(f.aux.p[(lr.sel >> 1) & 1] + at, w);
        const u64* add = f.add.p[(lr.sel >> 1) & 1];
        if (add != nullptr) dag.set.read(add + at, w);
      }
    }
  }
  dag.commit();
  if (t.logn <= nttk::kWholeMaxLog) {
    prof_before(KID_NTT_SMALL);
    nttk::launch_whole<false>(in, out, b, t, c->stream, pro, epi, f.multi);
    prof_after(KID_NTT_SMALL, b.count);
    c->launches++;
    CUDA_CHECK(cudaGetLastError());
    return;
  }
  prof_before(KID_NTT_STRIDED);
  nttk::launch_strided<false>(in, ptr2(mid), b1, n_int, t, c->stream, pro);
  prof_after(KID_NTT_STRIDED, b.count);
  prof_before(KID_NTT_CONTIG);
  nttk::launch_contig<false>(ptr2(mid), out, b2, n_int, t, c->stream, epi, f.multi);
  prof_after(KID_NTT_CONTIG, b.count);
  c->launches += 2;
  CUDA_CHECK(cudaGetLastError());
}

void launch_ntt(Ptr2 in, Ptr2 out, const LimbBatch& b, bool inverse, const Twiddle* last) {
  if (b.count == 0) return;
  if (inverse)
    launch_dir<true>(in, out, b, last);
  else
    launch_dir<false>(in, out, b, nullptr);
}

}  // namespace fhert
