// Per-pixel sample streams on the device: Z-Sobol index permutation, Owen-
// scrambled Sobol (Laine-Karras) and the PCG hash, integer-exact restatement of
// crates/renderer/src/sampler/{pcg,zsobol,aux_rng,path_sampler}.rs.
#pragma once
#include <cstdint>

namespace tpt {

__device__ __forceinline__ uint32_t pcg_state_transition(uint32_t s) { return s * 747796405u + 2891336453u; }
__device__ __forceinline__ uint32_t pcg_output(uint32_t s) {
  s ^= s >> (4u + (s >> 28));
  s *= 277803737u;
  return s ^ (s >> 22);
}
__device__ __forceinline__ uint32_t pcg_hash(uint32_t k) { return pcg_output(pcg_state_transition(k)); }

__device__ __forceinline__ uint32_t lk_permutation(uint32_t v, uint32_t seed) {
  v ^= v * 0x3d20adeau;
  v += seed;
  v *= (seed >> 16) | 1u;
  v ^= v * 0x05526c56u;
  v ^= v * 0x53a22864u;
  return v;
}

__device__ __forceinline__ float uint_to_float(uint32_t v) {
  const uint32_t mask = v >> 24;
  return __uint2float_rn(v & ~mask) * (1.0f / 4294967296.0f);
}

__device__ __forceinline__ uint64_t mix_bits(uint64_t v) {
  v ^= v >> 31;
  v *= 0x7fb5d329728ea185ull;
  v ^= v >> 27;
  v *= 0x81dadef4bc2dd44dull;
  v ^= v >> 33;
  return v;
}

__device__ __forceinline__ uint64_t left_shift_2(uint64_t v) {
  v &= 0xffffffffull;
  v = (v ^ (v << 16)) & 0x0000ffff0000ffffull;
  v = (v ^ (v << 8)) & 0x00ff00ff00ff00ffull;
  v = (v ^ (v << 4)) & 0x0f0f0f0f0f0f0f0full;
  v = (v ^ (v << 2)) & 0x3333333333333333ull;
  v = (v ^ (v << 1)) & 0x5555555555555555ull;
  return v;
}

// zsobol.rs:98-171, the first two generator matrices (no draw is wider than
// 2D).  Dimension 0 reverses the bits.  Dimension 1 is the Pascal matrix: input
// bit i feeds output bit j iff i & j == 0, so the output is the GF(2) sum over
// the subsets of ~j: four shift-and-xor steps, then a bit reversal (~j).
__device__ __forceinline__ uint32_t sobol_reversed_0(uint32_t index16) { return __brev(index16) >> 16; }
__device__ __forceinline__ uint32_t sobol_reversed_1(uint32_t index16) {
  uint32_t z = index16;
  z ^= (z & 0x5555u) << 1;
  z ^= (z & 0x3333u) << 2;
  z ^= (z & 0x0F0Fu) << 4;
  z ^= (z & 0x00FFu) << 8;
  return __brev(z) >> 16;
}

// zsobol.rs:238-263: the 24 permutations of a base-4 digit, one byte each
// (2 bits per digit: permutation p maps digit d to (byte_p >> 2d) & 3), packed
// into three 64-bit immediates so a per-lane index costs ALU work instead of a
// serialized constant-bank access.
__device__ __forceinline__ uint32_t perm_digit(uint32_t p, uint32_t digit) {
  uint64_t w;
  if (p < 8) w = 0xB1E19C6C78D8B4E4ull;        // p 0..7:  E4 B4 D8 78 6C 9C E1 B1
  else if (p < 16) w = 0x72D236C68D2D39C9ull;  // p 8..15: C9 39 2D 8D C6 36 D2 72
  else w = 0x93634B1B87271E4Eull;              // p 16..23: 4E 1E 27 87 1B 4B 63 93
  const uint32_t byte = (uint32_t)(w >> (8u * (p & 7u))) & 0xFFu;
  return (byte >> (2u * digit)) & 3u;
}

// The index permutation for Morton indices of at most 32 bits (image side^2 x
// spp up to 2^32: 1080p at 1,024 spp, 4096^2 at 256), in 32-bit arithmetic.
// The draws are most of a shading vertex's instructions (a 256 x 256 x 64 image
// has 11 digits per draw, four to six draws per vertex), so the digit step is
// written for instruction count; its value is mix_bits' bit for bit:
//  - `higher` is below 2^30, so bit 31 and the high word of higher ^ dim_hash
//    are the dimension's: the first xor-shift and the high word's share of the
//    first product are per-dimension constants (DimHash);
//  - bits 24.. of the mixed value modulo 24 = 8 (bits 27.. mod 3) + bits 24-26:
//    256 = 1 (mod 3), so a byte sum (dp4a) leaves at most 2,071 to reduce;
//  - table T_d holds permutation p's image of digit d in bits 2p, and
//    T_3 = T_0 ^ T_1 ^ T_2 (a permutation's images are 0..3), so a digit picks
//    its table with two masked xors; the table serves every dimension drawn.
// Measured against the 64-bit digit loop (a 64-bit modulo by 24 and a 64-bit
// variable shift per digit), with draws nobody reads left out: Cornell box
// 256 x 256 x 64 11.71 -> 10.44 ms, the 2.1M-triangle scene 1080p x 16
// 115.8 -> 106.9 ms.
struct DimHash {
  uint32_t x, k;
};
constexpr uint32_t kMix1Lo = 0x728ea185u, kMix1Hi = 0x7fb5d329u, kMix2Lo = 0xbc2dd44du, kMix2Hi = 0x81dadef4u;
__device__ __forceinline__ DimHash dim_hash32(uint32_t dimension) {
  const uint64_t h = 0x55555555ull * (uint64_t)dimension;
  const uint32_t lo = (uint32_t)h, hi = (uint32_t)(h >> 32);
  return DimHash{lo ^ ((hi << 1) | (lo >> 31)), (hi ^ (hi >> 31)) * kMix1Lo};
}
// mix_bits(higher ^ dim_hash) for higher < 2^31: low and high word
__device__ __forceinline__ void mix_bits32(uint32_t higher, DimHash h, uint32_t& lo, uint32_t& hi) {
  const uint32_t v = higher ^ h.x;
  const uint64_t p = (uint64_t)v * kMix1Lo + ((uint64_t)h.k << 32);
  const uint32_t p_lo = (uint32_t)p, p_hi = (uint32_t)(p >> 32) + v * kMix1Hi;
  const uint32_t v_lo = p_lo ^ ((p_hi << 5) | (p_lo >> 27)), v_hi = p_hi ^ (p_hi >> 27);
  const uint64_t q = (uint64_t)v_lo * kMix2Lo;
  hi = (uint32_t)(q >> 32) + v_lo * kMix2Hi + v_hi * kMix2Lo;
  lo = (uint32_t)q ^ (hi >> 1);
}
template <int N>
__device__ __forceinline__ void sample_index32(uint32_t morton, uint32_t log2_spp, uint32_t n_digits,
                                               const uint32_t (&dim)[N], uint32_t (&out)[N]) {
  DimHash h[N];
#pragma unroll
  for (int k = 0; k < N; ++k) {
    h[k] = dim_hash32(dim[k]);
    out[k] = 0;
  }
  const uint32_t odd = log2_spp & 1u;
  uint32_t shift = 2u * n_digits - odd;  // bits of the index not yet permuted
  // the top digit has no digits above it: `higher` starts at 0, and the shift
  // below never reaches 32
  uint32_t higher = 0;
#pragma unroll 2
  for (; shift > odd; shift -= 2u) {
    const uint32_t rest = morton >> (shift - 2u);
    const uint32_t m1 = 0u - (rest & 1u), m2 = 0u - ((rest >> 1) & 1u);
    const uint32_t t_lo = 0xaa555000u ^ (m1 & 0xafaf5fa5u) ^ (m2 & 0x7679b6deu);
    const uint32_t t_hi = 0x0000fffau ^ (m1 & 0x0000f5a5u) ^ (m2 & 0x00009edeu);
#pragma unroll
    for (int k = 0; k < N; ++k) {
      uint32_t lo, hi;
      mix_bits32(higher, h[k], lo, hi);
      const uint32_t s = __dp4a(hi, 0x02020202u, lo >> 27);
      const uint32_t q = (s * 0x5556u) >> 16;  // s / 3
      // halfword s % 3 of the table, then pair (bits 24-26) of its eight
      const uint32_t half = __byte_perm(t_lo, t_hi, s * 0x22u + 0x10u - q * 0x66u);
      out[k] = out[k] * 4u + ((half >> ((lo >> 23) & 14u)) & 3u);
    }
    higher = rest;
  }
  if (odd) {
#pragma unroll
    for (int k = 0; k < N; ++k) {
      uint32_t lo, hi;
      mix_bits32(morton >> 1, h[k], lo, hi);
      out[k] = out[k] * 2u + ((morton ^ lo) & 1u);
    }
  }
}

// IndexSampler (zsobol.rs:206-285) + PathSampler (path_sampler.rs:146-250).
// ANY: the pixel and sample may lie outside the image, whose Morton index can be
// longer than the image's digits; a digit's permutation depends on every bit above
// it, so such an index takes the 64-bit loop.  Render paths lie inside by
// construction and leave the check out.
template <bool ANY>
struct PathSampler {
  uint64_t morton;  // (encode_morton_2(px, py) << log2_spp) | sample
  uint32_t log2_spp;
  uint32_t n_base4_digits;
  uint32_t seed;  // the scramble seed: 0 is the reference's SCRAMBLE_SEED (path_sampler.rs:77)

  __device__ __forceinline__ void init(uint32_t px, uint32_t py, uint32_t sample, uint32_t log2spp, uint32_t ndig,
                                       uint32_t scramble = 0u) {
    log2_spp = log2spp;
    n_base4_digits = ndig;
    seed = scramble;
    morton = (((left_shift_2(py) << 1) | left_shift_2(px)) << log2spp) | (uint64_t)sample;
  }

  __device__ __forceinline__ uint64_t sample_index(uint32_t dimension) const {
    uint64_t out = 0;
    const bool pow2 = (log2_spp & 1u) != 0;
    const int last = pow2 ? 1 : 0;
    const uint64_t dim_hash = 0x55555555ull * (uint64_t)dimension;
    for (int i = (int)n_base4_digits - 1; i >= last; --i) {
      const uint32_t shift = 2u * (uint32_t)i - (pow2 ? 1u : 0u);
      const uint32_t digit = (uint32_t)((morton >> shift) & 3u);
      const uint64_t higher = morton >> (shift + 2);
      const uint32_t p = (uint32_t)((mix_bits(higher ^ dim_hash) >> 24) % 24u);
      out |= (uint64_t)perm_digit(p, digit) << shift;
    }
    if (pow2) out |= (morton & 1u) ^ (mix_bits((morton >> 1) ^ dim_hash) & 1u);
    return out;
  }

  __device__ __forceinline__ bool narrow() const {
    const uint32_t bits = 2u * n_base4_digits - (log2_spp & 1u);
    return bits <= 32u && (!ANY || (morton >> bits) == 0);
  }

  // sample_index of N dimensions, its words folded by xor
  template <int N>
  __device__ __forceinline__ void folded_indices(const uint32_t (&dim)[N], uint32_t (&index)[N]) const {
    if (narrow()) {
      sample_index32<N>((uint32_t)morton, log2_spp, n_base4_digits, dim, index);
    } else {
#pragma unroll
      for (int k = 0; k < N; ++k) {
        const uint64_t si = sample_index(dim[k]);
        index[k] = (uint32_t)si ^ (uint32_t)(si >> 32);
      }
    }
  }
  // the Owen-scrambled Sobol point of a dimension at a folded index
  template <bool SECOND>
  __device__ __forceinline__ void point(uint32_t dimension, uint32_t index, float& a, float& b) const {
    const uint64_t sb = mix_bits(((uint64_t)this->seed << 32) | (uint64_t)dimension);  // seed_for_dimension
    const uint32_t seed = (uint32_t)sb ^ (uint32_t)(sb >> 32);
    const uint32_t idx = lk_permutation(__brev(index), seed) >> 16;
    a = uint_to_float(__brev(lk_permutation(sobol_reversed_0(idx), seed)));
    if (SECOND) b = uint_to_float(__brev(lk_permutation(sobol_reversed_1(idx), (seed >> 8) | (seed << 24))));
  }
  // Out of line and by value: a draw is some 400 instructions, and a shading
  // vertex makes several; the kernels keep one copy of each form.
  static __device__ __noinline__ float draw_1(PathSampler s, uint32_t dim) {
    const uint32_t d[1] = {dim};
    uint32_t i[1];
    s.folded_indices<1>(d, i);
    float a, b;
    s.point<false>(dim, i[0], a, b);
    return a;
  }
  static __device__ __noinline__ float2 draw_2(PathSampler s, uint32_t dim) {
    const uint32_t d[1] = {dim};
    uint32_t i[1];
    s.folded_indices<1>(d, i);
    float2 r;
    s.point<true>(dim, i[0], r.x, r.y);
    return r;
  }
  // a 2D and a 1D draw (z) of one vertex together: the digit's share of the work
  // once, and two independent chains for the scheduler
  static __device__ __noinline__ float3 draw_21(PathSampler s, uint32_t dim2, uint32_t dim1) {
    const uint32_t d[2] = {dim2, dim1};
    uint32_t i[2];
    s.folded_indices<2>(d, i);
    float3 r;
    float unused;
    s.point<true>(dim2, i[0], r.x, r.y);
    s.point<false>(dim1, i[1], r.z, unused);
    return r;
  }
  // 1D draws of four consecutive dimensions
  static __device__ __noinline__ float4 draw_1111(PathSampler s, uint32_t dim) {
    const uint32_t d[4] = {dim, dim + 1u, dim + 2u, dim + 3u};
    uint32_t i[4];
    s.folded_indices<4>(d, i);
    float4 r;
    float unused;
    s.point<false>(d[0], i[0], r.x, unused);
    s.point<false>(d[1], i[1], r.y, unused);
    s.point<false>(d[2], i[2], r.z, unused);
    s.point<false>(d[3], i[3], r.w, unused);
    return r;
  }
  __device__ __forceinline__ float4 sample_1d4(uint32_t first_dim) const { return draw_1111(*this, first_dim); }
  __device__ __forceinline__ float sample_1d(uint32_t dim) const { return draw_1(*this, dim); }
  __device__ __forceinline__ void sample_2d(uint32_t dim, float& a, float& b) const {
    const float2 r = draw_2(*this, dim);
    a = r.x;
    b = r.y;
  }
  __device__ __forceinline__ void sample_2d_1d(uint32_t dim2, uint32_t dim1, float& a, float& b, float& c) const {
    const float3 r = draw_21(*this, dim2, dim1);
    a = r.x;
    b = r.y;
    c = r.z;
  }
  __device__ __forceinline__ uint32_t aux_rng_seed(uint32_t dim) const {
    uint64_t si;
    if (narrow()) {
      const uint32_t d[1] = {dim};
      uint32_t i[1];
      sample_index32<1>((uint32_t)morton, log2_spp, n_base4_digits, d, i);
      si = i[0];
    } else {
      si = sample_index(dim);
    }
    const uint64_t bits = mix_bits(si ^ ((uint64_t)dim << 32) ^ (uint64_t)seed);
    return pcg_hash((uint32_t)bits ^ (uint32_t)(bits >> 32));
  }
};
using PathSamplerDev = PathSampler<false>;

// Dimension layout (path_sampler.rs:153-169): camera at 0, vertex `depth` at
// 2 + 16 * depth + offset.
constexpr uint32_t kDimCamera = 0;
__device__ __forceinline__ uint32_t vertex_dim(uint32_t depth, uint32_t offset) { return 2u + 16u * depth + offset; }
constexpr uint32_t kOffCategory = 0, kOffTree = 1, kOffLightAux = 2, kOffSurface = 3, kOffLobe = 5, kOffLayer = 6,
                   kOffDir = 7, kOffExtra0 = 9, kOffExtra1 = 10, kOffExtra2 = 11, kOffExtra3 = 12, kOffRr = 13,
                   kOffAuxSeed = 14;

}  // namespace tpt
