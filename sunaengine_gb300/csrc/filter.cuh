// Candidate filter of the list builds: byte-coded places tested against one's
// own with an add and a byte dot product, four candidates to a 16-byte load. What
// the codes and bounds are, and why no neighbour is dropped, stands at each user
// (sim2d.cuh, sim3d.cuh).
#pragma once
#include <cstdint>

namespace sn {

// Bounds on the dot product, for accumulators that go negative: `far` drops a
// candidate, `near` accepts it without the exact test.
struct CandBounds {
  int32_t far, near;
};
// Candidates [base, base + 32) that lie in [lo, hi), base a multiple of 4, as two
// masks with candidate base + j at bit 31 - j: the survivors, and those of them
// near enough to need no test. NV vectors are in flight.
struct CandMask {
  uint32_t hit, near;
};
template <int NV>
__device__ __forceinline__ CandMask cand_mask(const uint32_t* QC, uint32_t base, uint32_t lo, uint32_t hi,
                                              uint32_t bias, CandBounds cb) {
  const uint32_t nv = min((hi - base + 3u) >> 2, 8u);
  const uint4* src = reinterpret_cast<const uint4*>(QC + base);
  const int32_t step = cb.near - cb.far;
  CandMask m{0u, 0u};
  auto test = [&](uint32_t code) {
    const int d = (int)(code + bias);
    const int32_t acc = __dp4a(d, d, cb.far);
    m.hit = __funnelshift_l((uint32_t)acc, m.hit, 1);
    m.near = __funnelshift_l((uint32_t)(acc + step), m.near, 1);
  };
  for (uint32_t v = 0; v < nv; v += NV) {
    uint4 w[NV];
#pragma unroll
    for (int j = 0; j < NV; ++j) w[j] = src[min(v + j, nv - 1u)];
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      test(w[j].x);
      test(w[j].y);
      test(w[j].z);
      test(w[j].w);
    }
  }
  // codes shifted in so far (a repeated vector's lie past hi), to the top; the
  // ones outside [lo, hi) dropped
  const uint32_t done = 4u * ((nv + NV - 1u) / NV * NV);
  uint32_t in = 0xffffffffu << (32u - done);
  if (lo > base) in &= 0xffffffffu >> (lo - base);
  if (hi - base < 32u) in &= ~(0xffffffffu >> (hi - base));
  m.hit = (m.hit << (32u - done)) & in;
  m.near = m.near << (32u - done);
  return m;
}

}  // namespace sn
