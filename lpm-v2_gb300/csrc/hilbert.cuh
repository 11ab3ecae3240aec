// hilbert.cuh -- index along a Hilbert curve of a cell of a 2^16 x 2^16 grid (2-D), of a direction on
// the cube around the sphere, and of a cell of a 2^10 x 2^10 x 2^10 grid (3-D; the orders below do
// not use it: where that curve leaves the sphere's shell and enters it again elsewhere, consecutive
// sources lie in two pieces).
//
// J. Skilling, "Programming the Hilbert curve", AIP Conf. Proc. 707, 381 (2004): the cell
// coordinates are turned in place into the "transpose" of the Hilbert index (undo the
// excess rotations and reflections level by level, then Gray-encode), and the index is the
// bitwise interleave of the three transposed words, most significant bit of axis 0 first.
#pragma once

#include <cstdint>

namespace lpm {

// Bits 0..9 of v moved to bits 0, 3, 6, ..., 27.
__host__ __device__ inline uint32_t spread10(uint32_t v) {
  v &= 0x3ffu;
  v = (v | (v << 16)) & 0x030000ffu;
  v = (v | (v << 8)) & 0x0300f00fu;
  v = (v | (v << 4)) & 0x030c30c3u;
  v = (v | (v << 2)) & 0x09249249u;
  return v;
}

__host__ __device__ inline uint32_t hilbert_index30(uint32_t x0, uint32_t x1, uint32_t x2) {
  uint32_t X[3] = {x0 & 0x3ffu, x1 & 0x3ffu, x2 & 0x3ffu};
  for (uint32_t q = 1u << 9; q > 1u; q >>= 1) {
    const uint32_t p = q - 1u;
    for (int i = 0; i < 3; ++i) {
      if (X[i] & q) {
        X[0] ^= p;  // invert the lower bits of axis 0
      } else {
        const uint32_t t = (X[0] ^ X[i]) & p;  // exchange the lower bits of axes 0 and i
        X[0] ^= t;
        X[i] ^= t;
      }
    }
  }
  X[1] ^= X[0];
  X[2] ^= X[1];
  uint32_t t = 0;
  for (uint32_t q = 1u << 9; q > 1u; q >>= 1) {
    if (X[2] & q) t ^= q - 1u;
  }
  X[0] ^= t;
  X[1] ^= t;
  X[2] ^= t;
  return (spread10(X[0]) << 2) | (spread10(X[1]) << 1) | spread10(X[2]);
}

// Bits 0..15 of v moved to bits 0, 2, 4, ..., 30.
__host__ __device__ inline uint32_t spread16(uint32_t v) {
  v &= 0xffffu;
  v = (v | (v << 8)) & 0x00ff00ffu;
  v = (v | (v << 4)) & 0x0f0f0f0fu;
  v = (v | (v << 2)) & 0x33333333u;
  v = (v | (v << 1)) & 0x55555555u;
  return v;
}

// The same construction in two dimensions, 16 bits per axis.
__host__ __device__ inline uint32_t hilbert_index2d(uint32_t x0, uint32_t x1) {
  uint32_t X[2] = {x0 & 0xffffu, x1 & 0xffffu};
  for (uint32_t q = 1u << 15; q > 1u; q >>= 1) {
    const uint32_t p = q - 1u;
    for (int i = 0; i < 2; ++i) {
      if (X[i] & q) {
        X[0] ^= p;
      } else {
        const uint32_t t = (X[0] ^ X[i]) & p;
        X[0] ^= t;
        X[i] ^= t;
      }
    }
  }
  X[1] ^= X[0];
  uint32_t t = 0;
  for (uint32_t q = 1u << 15; q > 1u; q >>= 1) {
    if (X[1] & q) t ^= q - 1u;
  }
  X[0] ^= t;
  X[1] ^= t;
  return (spread16(X[0]) << 1) | spread16(X[1]);
}

// The curve index of a point's direction, of `bits` bits (3 + 2 k): the six faces of the cube around
// the sphere in turn, on each a 2-D Hilbert curve over 2^k x 2^k cells, laid so that one face's
// curve ends at the cube's corner where the next one's starts.  The faces' gnomonic coordinates are
// evened out by u (1.273 - 0.273 |u|), about (4 / pi) atan u.  Groups of 32 of 98,304 even sources have a
// mean radius of 0.052 (95 % below 0.067) in this order, 0.076 (0.159) along the 3-D curve.
constexpr int kSphereCurveBits = 23;      // three passes of a radix sort
constexpr int kSphereCurveBitsFine = 27;  // four

__host__ __device__ inline uint32_t sphere_curve_index(float x, float y, float z, int bits) {
  const float ax = x < 0.f ? -x : x, ay = y < 0.f ? -y : y, az = z < 0.f ? -z : z;
  uint32_t face;
  float m, u, v;  // the largest component, and the face's coordinates along and across its curve
  if (ax >= ay && ax >= az) {
    m = ax;
    face = x < 0.f ? 0u : 5u;
    u = x < 0.f ? z : -y;
    v = x < 0.f ? y : -z;
  } else if (ay >= az) {
    m = ay;
    face = y < 0.f ? 1u : 3u;
    u = y < 0.f ? -z : z;
    v = x;
  } else {
    m = az;
    face = z < 0.f ? 2u : 4u;
    u = z < 0.f ? y : x;
    v = z < 0.f ? x : -y;
  }
  const float inv = m > 0.f ? 1.f / m : 0.f;
  uint32_t c[2];
  for (int k = 0; k < 2; ++k) {
    const float w = (k == 0 ? u : v) * inv, wa = w < 0.f ? -w : w;
    const float q = (w * (1.273f - 0.273f * wa) + 1.f) * 32768.f;
    c[k] = q > 0.f ? (q < 65535.f ? static_cast<uint32_t>(q) : 65535u) : 0u;  // (NaN: 0)
  }
  return (face << (bits - 3)) | (hilbert_index2d(c[0], c[1]) >> (35 - bits));
}

}  // namespace lpm
