// Client-side entry points of the C ABI: seeding, encode, encrypt, decrypt,
// decode and key export.  Citations name files inside fhe-cmplr/rtlib/ant/.
#include <algorithm>
#include <cmath>
#include <complex>
#include <cstring>
#include <vector>

#include "runtime.h"

using namespace fhert;

namespace {

typedef std::complex<double> cplx;

constexpr int64_t kMax64 = (int64_t)(((u64)1 << 63) - ((u64)1 << 9)) - 1;

uint32_t reverse_bits(uint32_t v, int bits) {
  uint32_t r = 0;
  for (int i = 0; i < bits; i++) r |= ((v >> i) & 1u) << (bits - 1 - i);
  return r;
}

// util/src/ntt.c:562-590: roots e^(2 pi i k / 2N) and the powers of 5 mod 2N
void ensure_fft_tables(Context* c) {
  if (!c->fft_rou_re.empty()) return;
  size_t m = 2ull * c->N;
  c->fft_rou_re.resize(m);
  c->fft_rou_im.resize(m);
  for (size_t i = 0; i < m; i++) {
    double angle     = 2 * M_PI * i / m;
    c->fft_rou_re[i] = std::cos(angle);
    c->fft_rou_im[i] = std::sin(angle);
  }
  size_t slots = c->N / 2;
  c->fft_rot_group.resize(slots);
  c->fft_rot_group[0] = 1;
  for (size_t i = 1; i < slots; i++)
    c->fft_rot_group[i] = (uint32_t)((5ull * c->fft_rot_group[i - 1]) % m);
}

// complex product with the textbook formula and separately rounded operations,
// as the C compiler of the CPU runtime evaluates it
inline cplx cmul(cplx a, cplx b) {
  double re = a.real() * b.real() - a.imag() * b.imag();
  double im = a.real() * b.imag() + a.imag() * b.real();
  return cplx(re, im);
}

// util/src/ntt.c:633-675
void embedding_inv(Context* c, std::vector<cplx>& v) {
  size_t len = v.size(), m = 2ull * c->N;
  int    lg  = 0;
  while ((1ull << lg) < len) lg++;
  for (int logm = lg; logm > 0; logm--) {
    size_t idx_mod = 1ull << (logm + 2), gap = m / idx_mod, num1 = 1ull << logm,
           num2 = 1ull << (logm - 1);
    for (size_t j = 0; j < len; j += num1) {
      for (size_t i = 0; i < num2; i++) {
        size_t e = j + i, o = j + i + num2;
        size_t r = (idx_mod - (c->fft_rot_group[i] % idx_mod)) * gap;
        cplx   plus = v[e] + v[o], minus = v[e] - v[o];
        minus = cmul(minus, cplx(c->fft_rou_re[r], c->fft_rou_im[r]));
        v[e]  = plus;
        v[o]  = minus;
      }
    }
  }
  std::vector<cplx> out(len);
  for (size_t i = 0; i < len; i++) out[i] = v[reverse_bits((uint32_t)i, lg)];
  double d = (double)len;
  for (size_t i = 0; i < len; i++) v[i] = cplx(out[i].real() / d, out[i].imag() / d);
}

void init_plain(Context* c, PLAIN plain, size_t level, double scale, uint32_t sf_degree,
                uint32_t slots = 0, size_t num_p = 0) {
  POLY p = &plain->_poly;
  // special limbs sit at the end of the allocation, so an extended plaintext
  // needs storage of exactly level + K limbs
  if (p->_data == nullptr || (num_p ? p->_num_alloc_primes != level + num_p
                                    : p->_num_alloc_primes < level)) {
    Free_poly_data(p);
    Alloc_poly_data(p, c->N, level, num_p);
  } else {
    p->_num_primes   = level;
    p->_num_primes_p = num_p;
  }
  plain->_scaling_factor = scale;
  plain->_sf_degree      = sf_degree;
  plain->_slots          = slots ? slots : c->N / 2;
}

// level Q limbs, then num_p special limbs stored right behind them
LimbBatch q_batch(size_t level, size_t num_p = 0, int first_p_prime = 0) {
  LimbBatch b;
  b.count = (int)(level + num_p);
  for (size_t i = 0; i < level; i++)
    b.limb[i] = LimbRef{(uint16_t)i, (uint16_t)i, (uint16_t)i, (uint8_t)i, 0};
  for (size_t k = 0; k < num_p; k++) {
    uint16_t at = (uint16_t)(level + k);
    b.limb[level + k] = LimbRef{at, at, at, (uint8_t)(first_p_prime + k), 0};
  }
  return b;
}

}  // namespace

namespace fhert {

// ckks/src/encoder.c:473-520: residues of one real value at the given scale,
// on level Q limbs followed by num_p special limbs
std::vector<int64_t> encode_value(Context* c, double value, uint32_t level, double scale,
                                  uint32_t num_p) {
  FHERT_ASSERT(level > 0 && level <= (uint32_t)c->L, "level should not be larger than q_cnt");
  FHERT_ASSERT(num_p == 0 || num_p == (uint32_t)c->K, "invalid p cnt");
  int32_t log_scale  = (int32_t)std::log2(std::fabs(value * scale));
  int32_t log_valid  = log_scale <= 61 ? log_scale : 61;
  int32_t log_approx = log_scale - log_valid;
  double  scaled     = value / std::pow(2, log_approx) * scale;
  int64_t val_int    = (int64_t)scaled;
  std::vector<int64_t> res(level + num_p);
  for (uint32_t i = 0; i < level + num_p; i++) {
    int64_t q = (int64_t)c->primes[i < level ? i : c->L + (i - level)], r = val_int % q;
    res[i] = r < 0 ? r + q : r;
  }
  if (log_approx > 0) {
    // scale back up by 2^log_approx in steps of at most 61 then 60 bits
    for (uint32_t i = 0; i < level; i++) {
      u64     q = c->primes[i];
      int32_t left = log_approx, step = left <= 61 ? left : 61;
      u64     f = (1ull << step) % q;
      left -= step;
      while (left > 0) {
        step = left <= 60 ? left : 60;
        f    = mulmod(f, (1ull << step) % q, q);
        left -= step;
      }
      res[i] = (int64_t)mulmod((u64)res[i], f, q);
    }
  }
  return res;
}

// ckks/src/encoder.c:234-325; slots = 0 means N/2, num_p = K also fills the
// special limbs (the plaintexts of the bootstrapping linear transforms)
void encode_vector(Context* c, PLAIN plain, const MessageInput& in, uint32_t sf_degree,
                   uint32_t level, uint32_t slots, uint32_t num_p) {
  LaunchScope    scope;
  const uint32_t n = c->N;
  if (slots == 0) slots = n / 2;
  FHERT_ASSERT(slots <= n / 2 && (slots & (slots - 1)) == 0, " slot size > N/2 ");
  FHERT_ASSERT(num_p == 0 || num_p == (uint32_t)c->K, "invalid p cnt");
  if (level == 0) level = c->L;
  FHERT_ASSERT(level <= (uint32_t)c->L, "level should not be larger than mul_depth + 1");
  FHERT_ASSERT(in.count <= slots, "slot size is too small");
  FHERT_ASSERT(sf_degree >= 1, "invalid scaling factor for encode");
  const double delta = std::pow(2.0, (double)c->sf_bits);
  init_plain(c, plain, level, std::pow(delta, (double)sf_degree), sf_degree, slots, num_p);
  int64_t* d_msg = nullptr;
  CUDA_CHECK(dev_alloc(&d_msg, n * sizeof(int64_t), c->stream));
  // inverse embedding, scaling and rounding run on the device with the host
  // routine's arithmetic (embedding.cu)
  encode_message_on_device(c, in, slots, d_msg);
  message_to_ntt(c, plain->_poly._data, d_msg, 1, sf_degree > 1 ? scale_powers(c, sf_degree) : nullptr,
                 q_batch(level, num_p, c->L));
  CUDA_CHECK(dev_free(d_msg, c->stream));
  plain->_poly._is_ntt = true;
}

}  // namespace fhert

namespace {

// ckks/src/encoder.c:473-575: one value on every coefficient of every limb
void encode_scalar(Context* c, PLAIN plain, double value, uint32_t sf_degree, uint32_t level) {
  LaunchScope scope;
  if (level == 0) level = c->L;
  const double delta = std::pow(2.0, (double)c->sf_bits), scale = std::pow(delta, sf_degree);
  init_plain(c, plain, level, scale, sf_degree);
  std::vector<int64_t> res = encode_value(c, value, level, scale, 0);
  // fill every limb with its residue: one clear, one launch for all limbs
  POLY p = &plain->_poly;
  CUDA_CHECK(zero_async(p->_data, (size_t)level * c->N * sizeof(int64_t), c->stream));
  std::vector<u64> sc(res.begin(), res.end());
  launch_scalars(false, ptr2(p->_data), ptr2(p->_data), sc.data(), q_batch(level));
  p->_is_ntt = true;
}

}  // namespace

extern "C" {

void Fhert_seed(const uint32_t seed[16], uint64_t counter, int64_t fake_time_us) {
  seed_prng(seed, counter, fake_time_us);
}

// ckks/src/cipher.c:172-186: would msg still fit the modulus at the
// ciphertext's level and scale
bool Within_value_range(CIPHER ciph, double* msg, uint32_t len) {
  Context* c     = ctx();
  uint32_t slots = ciph->_slots;
  FHERT_ASSERT(len <= slots, "length of msg should less than slots");
  ensure_fft_tables(c);
  std::vector<cplx> v(slots, cplx(0, 0));
  for (uint32_t i = 0; i < len; i++) v[i] = cplx(msg[i], 0.0);
  embedding_inv(c, v);
  double top = 0.0;
  for (auto& x : v) {
    top = std::max(top, std::fabs(x.real() * ciph->_scaling_factor));
    top = std::max(top, std::fabs(x.imag() * ciph->_scaling_factor));
  }
  int32_t bits  = (int32_t)std::log2(std::max(top, 2.2250738585072014e-308)) + 1;
  int32_t valid = (int32_t)c->q0_bits + ((int32_t)ciph->_c0_poly._num_primes - 1) * (int32_t)c->sf_bits;
  return bits < valid;
}

void Free_plain_data(PLAIN plain) { Free_poly_data(&plain->_poly); }

void Encode_double(PLAIN plain, double* input, size_t len, uint32_t sc_degree, uint32_t level) {
  Context* c = ctx();
  if (len == 1) {
    encode_scalar(c, plain, *input, sc_degree, level);
    return;
  }
  encode_vector(c, plain, MessageInput{MessageInput::kReals, input, len}, sc_degree, level);
}

void Encode_float(PLAIN plain, float* input, size_t len, uint32_t sc_degree, uint32_t level) {
  Context* c = ctx();
  if (len == 1) {
    encode_scalar(c, plain, (double)*input, sc_degree, level);
    return;
  }
  encode_vector(c, plain, MessageInput{MessageInput::kFloats, input, len}, sc_degree, level);
}

void Encode_dcmplx(PLAIN plain, double* re_im, size_t len, uint32_t sc_degree, uint32_t level) {
  encode_vector(ctx(), plain, MessageInput{MessageInput::kComplex, re_im, len}, sc_degree, level);
}

void Encode_double_mask(PLAIN plain, double cst, size_t len, uint32_t sc_degree, uint32_t level) {
  std::vector<double> m(len, cst);
  Encode_double(plain, m.data(), len, sc_degree, level);
}

void Encode_float_mask(PLAIN plain, float cst, size_t len, uint32_t sc_degree, uint32_t level) {
  std::vector<float> m(len, cst);
  Encode_float(plain, m.data(), len, sc_degree, level);
}

}  // extern "C"

// ---------------------------------------------------------------------------
// encrypt / decrypt / decode
// ---------------------------------------------------------------------------

extern "C" {

// ckks/src/encryptor.c:19-89
CIPHER Encrypt(CIPHER res, PLAIN plain) {
  LaunchScope scope;
  Context* c = ctx();
  FHERT_ASSERT(c->pk._p0._data != nullptr, "Encrypt: no public key (keys were not generated)");
  POLY   m     = &plain->_poly;
  size_t level = m->_num_primes;
  FHERT_ASSERT(m->_num_primes_p == 0, "Encrypt_msg: plain should not be extended");
  for (POLYNOMIAL* p : {&res->_c0_poly, &res->_c1_poly}) {
    if (p->_data == nullptr || p->_num_alloc_primes < level) {
      Free_poly_data(p);
      Alloc_poly_data(p, c->N, level, 0);
    } else {
      p->_num_primes   = level;
      p->_num_primes_p = 0;
    }
  }
  res->_scaling_factor = plain->_scaling_factor;
  res->_sf_degree      = plain->_sf_degree;
  res->_slots          = plain->_slots;
  if (!m->_is_ntt) Conv_poly2ntt_inplace(m);
  // u, e1, e2: triangle samples (small integers), sampled and transformed together
  int64_t *small = nullptr, *noise = nullptr;
  CUDA_CHECK(dev_alloc(&small, 3 * (size_t)c->N * sizeof(int64_t), c->stream));
  CUDA_CHECK(dev_alloc(&noise, 3 * level * c->N * sizeof(int64_t), c->stream));
  sample_triangles_on_device(c, small, 3);
  message_to_ntt(c, noise, small, 3, nullptr, q_batch(level));
  launch_encrypt(c, res->_c0_poly._data, res->_c1_poly._data, noise, m->_data, level);
  res->_c0_poly._is_ntt = res->_c1_poly._is_ntt = true;
  CUDA_CHECK(dev_free(small, c->stream));
  CUDA_CHECK(dev_free(noise, c->stream));
  return res;
}

// ckks/src/decryptor.c:19-66 (two-polynomial ciphertexts)
void Fhert_decrypt(PLAIN res, CIPHER ciph) {
  LaunchScope scope;
  Context* c     = ctx();
  size_t   level = ciph->_c0_poly._num_primes;
  FHERT_ASSERT(c->sk_ntt._data != nullptr, "Decrypt: no secret key");
  FHERT_ASSERT(ciph->_c0_poly._num_primes_p == 0, "Decrypt: ciph should not be extended");
  init_plain(c, res, level, ciph->_scaling_factor, ciph->_sf_degree);
  res->_slots    = ciph->_slots;
  // a ciphertext in coefficient form is brought to NTT form in place
  if (!ciph->_c1_poly._is_ntt) Conv_poly2ntt_inplace(&ciph->_c1_poly);
  if (!ciph->_c0_poly._is_ntt) Conv_poly2ntt_inplace(&ciph->_c0_poly);
  launch_decrypt(c, res->_poly._data, ciph->_c0_poly._data, ciph->_c1_poly._data, level);
  res->_poly._is_ntt = true;
}

// ckks/src/encoder.c:657-704: out receives `count` complex values as
// (re, im) pairs; the plaintext is left in coefficient form
void Fhert_decode(PLAIN plain, double* out, size_t count) {
  LaunchScope scope;
  Context* c = ctx();
  POLY           poly  = &plain->_poly;
  const uint32_t half  = c->N / 2;
  const uint32_t slots = plain->_slots ? plain->_slots : half;
  FHERT_ASSERT(count <= slots, "res size larger than decode size");
  if (poly->_is_ntt) Conv_ntt2poly_inplace(poly);
  decode_on_device(c, poly->_data, (int)poly->_num_primes, slots, plain->_scaling_factor, out, count);
}

// cipher.c Get_msg: decrypt and decode, real parts; the caller frees the result
double* Get_msg(CIPHER ciph) {
  PLAINTEXT plain;
  std::memset(&plain, 0, sizeof(plain));
  Fhert_decrypt(&plain, ciph);
  size_t              slots = plain._slots;
  std::vector<double> tmp(2 * slots);
  Fhert_decode(&plain, tmp.data(), slots);
  Free_poly_data(&plain._poly);
  double* out = (double*)std::malloc(slots * sizeof(double));
  for (size_t i = 0; i < slots; i++) out[i] = tmp[2 * i];
  return out;
}

// key material for inspection and parity checks: L Q limbs then K P limbs
void Fhert_export_switch_key(bool is_rot, int32_t rot_idx, uint32_t part, int which,
                             int64_t* host) {
  SW_KEY k = Swk(is_rot, rot_idx);
  POLY   p = which == 0 ? Pk0_at(k, part) : Pk1_at(k, part);
  Fhert_download(p, 0, p->_num_alloc_primes, host);
}

// which: 0 = secret key (coefficient form, L+K limbs), 1 = secret key in NTT
// form, 2 / 3 = public key polynomials (L limbs)
void Fhert_export_key(int which, int64_t* host) {
  Context* c = ctx();
  POLY     p = which == 0 ? &c->sk_s : which == 1 ? &c->sk_ntt : which == 2 ? &c->pk._p0 : &c->pk._p1;
  FHERT_ASSERT(p->_data != nullptr, "keys were not generated");
  Fhert_download(p, 0, p->_num_alloc_primes, host);
}

}  // extern "C"
