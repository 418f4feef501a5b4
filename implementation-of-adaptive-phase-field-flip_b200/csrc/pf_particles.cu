// Particle state between the caller's (n, 3) arrays and the float4 streams, one
// pass per direction.  The reference keeps plain arrays (pfflip/sim.py:142-155),
// so these passes have no counterpart there; they are bound by the bytes they
// move (60 B a particle in, 48 B out per array).  One thread a particle: the
// 16-byte side is fully coalesced, the 12-byte side is read or written in three
// words whose sectors the warp shares.
//
// Measured at 56.6 M particles against strided tensor copies and indexing:
// loading 2.2 -> 0.56 ms, reading both arrays back 2.9 -> 1.72 ms.
#include "pf_common.cuh"

namespace pf {

// pos4 = (x, y, z, liquid flag), vel4 = (u, v, w, index); either may be left out
__global__ void __launch_bounds__(256) k_pack(long long n, const float* __restrict__ pos,
                                              const int* __restrict__ type, float4* __restrict__ pos4,
                                              const float* __restrict__ vel, float4* __restrict__ vel4) {
  for (long long p = (long long)blockIdx.x * 256 + threadIdx.x; p < n; p += (long long)gridDim.x * 256) {
    if (pos4) {
      const float* x = pos + 3 * p;
      pos4[p] = make_float4(x[0], x[1], x[2], __int_as_float(type[p] == 1 ? PF_FLAG_LIQUID : 0));
    }
    if (vel4) {
      const float* v = vel + 3 * p;
      vel4[p] = make_float4(v[0], v[1], v[2], __int_as_float((int)p));
    }
  }
}

// rows of streams a4, b4 to their original places: out[index] = (x, y, z).  The
// destinations are scattered, so the pass is bound by the 32-byte sectors its
// stores touch in L2: a warp turns its 32 rows into 96 words and stores them 32
// at a time, three lanes to a row, instead of one word of 32 rows at a time (a
// third of the sectors; 1.99 -> 1.72 ms for both arrays at 56.6 M particles).
__global__ void __launch_bounds__(256) k_unpack(long long n, const float4* __restrict__ ids,
                                                const float4* __restrict__ a4, float* __restrict__ oa,
                                                const float4* __restrict__ b4, float* __restrict__ ob) {
  __shared__ float words[8][96];
  const int lane = threadIdx.x & 31;
  float* w = words[threadIdx.x >> 5];
  for (long long base = (long long)blockIdx.x * 256 + (threadIdx.x & ~31); base < n; base += (long long)gridDim.x * 256) {
    const long long p = base + lane;  // the loop is warp-uniform: every lane takes the shuffles
    const bool in = p < n;
    const int id = in ? __float_as_int(ids[p].w) : 0;
    const int rows = (int)(n - base < 32 ? n - base : 32);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      float* o = q ? ob : oa;
      if (!o) continue;
      if (in) {
        const float4 v = (q ? b4 : a4)[p];
        w[3 * lane] = v.x;
        w[3 * lane + 1] = v.y;
        w[3 * lane + 2] = v.z;
      }
      __syncwarp();
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const int e = 32 * k + lane, r = e / 3;
        const int rid = __shfl_sync(0xffffffffu, id, r);
        if (r < rows) o[3LL * rid + (e - 3 * r)] = w[e];
      }
      __syncwarp();
    }
  }
}

// the reverse gather: out4[p] = (in[index], 0); a missing input is zero
__global__ void __launch_bounds__(256) k_gather_rows(long long n, const float4* __restrict__ ids,
                                                     const float* __restrict__ a, float4* __restrict__ oa,
                                                     const float* __restrict__ b, float4* __restrict__ ob) {
  for (long long p = (long long)blockIdx.x * 256 + threadIdx.x; p < n; p += (long long)gridDim.x * 256) {
    const long long id = __float_as_int(ids[p].w);
    const float* x = a + 3 * id;
    oa[p] = a ? make_float4(x[0], x[1], x[2], 0.f) : make_float4(0.f, 0.f, 0.f, 0.f);
    const float* y = b + 3 * id;
    ob[p] = b ? make_float4(y[0], y[1], y[2], 0.f) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
}

int rows_grid(long long n) { return grid_for(n, 256, kNumSMs * 32); }

}  // namespace pf

using namespace pf;

extern "C" {

int pf_pack_particles(int64_t n, const float* pos, const int32_t* type, float* pos4, const float* vel, float* vel4,
                      void* stream) {
  PF_REQUIRE(n >= 0 && n < (1LL << 31), "bad particle count");
  if (n == 0) return PF_OK;
  PF_REQUIRE((pos4 || vel4) && (!pos4 || (pos && type)) && (!vel4 || vel), "null argument");
  PF_REQUIRE(aligned16(pos4) && aligned16(vel4), "particle streams must be 16-byte aligned");
  k_pack<<<rows_grid(n), 256, 0, S(stream)>>>(n, pos, type, reinterpret_cast<float4*>(pos4), vel,
                                              reinterpret_cast<float4*>(vel4));
  PF_LAUNCHED();
  return PF_OK;
}

int pf_unpack_particles(int64_t n, const float* vel4, const float* a4, float* a, const float* b4, float* b,
                        void* stream) {
  PF_REQUIRE(n >= 0, "bad particle count");
  if (n == 0) return PF_OK;
  PF_REQUIRE(vel4 && (a || b) && (!a || a4) && (!b || b4), "null argument");
  PF_REQUIRE(aligned16(vel4) && aligned16(a4) && aligned16(b4), "particle streams must be 16-byte aligned");
  k_unpack<<<rows_grid(n), 256, 0, S(stream)>>>(n, reinterpret_cast<const float4*>(vel4),
                                                reinterpret_cast<const float4*>(a4), a,
                                                reinterpret_cast<const float4*>(b4), b);
  PF_LAUNCHED();
  return PF_OK;
}

int pf_gather_particles(int64_t n, const float* vel4, const float* a, float* a4, const float* b, float* b4,
                        void* stream) {
  PF_REQUIRE(n >= 0, "bad particle count");
  if (n == 0) return PF_OK;
  PF_REQUIRE(vel4 && a4 && b4, "null argument");
  PF_REQUIRE(aligned16(vel4) && aligned16(a4) && aligned16(b4), "particle streams must be 16-byte aligned");
  k_gather_rows<<<rows_grid(n), 256, 0, S(stream)>>>(n, reinterpret_cast<const float4*>(vel4), a,
                                                     reinterpret_cast<float4*>(a4), b, reinterpret_cast<float4*>(b4));
  PF_LAUNCHED();
  return PF_OK;
}

}  // extern "C"
