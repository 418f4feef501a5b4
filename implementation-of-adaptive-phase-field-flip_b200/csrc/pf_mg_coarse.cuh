// The coarse end of the V-cycle in one launch of one CTA cluster: every level
// of up to about 80,000 cells (40^3 and below, any extents), pre-smoothing,
// residual and restriction on the way down, the coarsest solve, prolongation
// and post-smoothing on the way up (pfflip/poisson.py:312-345).
//
// What bounds it is the chain of half-sweeps, each a few hundred nanoseconds
// of work between two barriers, so everything is laid out to shorten a link:
//
// * A thread owns up to NQ quads of cells (k = 4h .. 4h + 3 of one row), two
//   of each colour, and keeps their face coefficients, omega/diagonal,
//   right-hand side and p in registers, as f32x2 pairs of one colour: a
//   half-sweep relaxes two cells per instruction.
// * p lives in two shared arrays, one per colour, indexed by (plane, row, k/2):
//   the neighbours of a red pair are a black pair at a fixed offset (one 8-byte
//   load, lanes on consecutive words), its neighbours along k are the thread's
//   own registers and one more word.  Walls need no tests: their coefficients
//   are zero and one halo plane on either side keeps every address inside.
// * A level of more than CC_NT * 2 quads (CC_NT * 3 for FP64 sweeps) is split into slabs of planes over the
//   cluster's CTAs; a thread that relaxes a boundary plane also stores its pair
//   into the neighbour's halo plane (st.async, counted on the neighbour's
//   mbarrier), so a half-sweep waits for its two neighbours and not for the
//   cluster (a cluster barrier of 16 CTAs takes 0.6 us).  A half-sweep reads
//   one colour and writes the other, so one halo copy is enough.  Smaller
//   levels run on one CTA, with CTA barriers only.
// * The levels from the first of at most kCcDenseMax cells down are one dense
//   operator, built with the hierarchy; its rows are spread over the cluster
//   and staged in shared memory, where they fit, before the right-hand side
//   exists.
// * Launched so that it may overlap the end of the kernel before it: the face
//   coefficients, the operator and the zeroed arrays are set up first.
//
// Measured on a B200, per V-cycle inside a solve, against one CTA holding the
// levels of up to 4096 cells (and an 8-CTA cluster where every extent is a
// multiple of 16) with launched sweeps above: 16^3 40 -> 18 us, 32^3 and below
// 52 -> 33 us, 24^3 (coarsest 6^3) 128 + 6 sweeps of 5 us -> 21 us, 30x22x18
// (coarsest 15x11x9 swept) 167 + 6 of 8 us -> 41 us, 31^3 swept 60 times
// 600 -> 62 us.  A half-sweep takes 0.5 us on one CTA (its shared-memory
// wavefronts are 0.2 us of that) and 0.7 us with the exchange.
//
// 16-bit hierarchies: storage is widened on load, p stays FP32 inside the
// kernel, the right-hand sides of the levels and the result are rounded to the
// storage type; the coarsest solve (sweeps on one CTA, or the dense operator)
// runs in FP64.  A swept coarsest level of more than 4096 cells, in slabs, is
// swept in FP32.
#pragma once

#include "pf_f32x2.cuh"

namespace pf {

constexpr int CC_NT = 512;        // threads per CTA
constexpr int CC_MAXC = 16;       // CTAs of the cluster
constexpr int kCcDenseMax = 512;  // cells of the largest level applied as a dense operator

// n / d for 0 <= n < 2^17 and d < 2^15, by one multiplication
struct CcDiv {
  unsigned mul;  // ceil(2^32 / d); 0 for d = 1
  __host__ __device__ __forceinline__ static CcDiv of(int d) {
    return CcDiv{d == 1 ? 0u : (unsigned)(((1ull << 32) + (unsigned)d - 1) / (unsigned)d)};
  }
  __device__ __forceinline__ int operator()(int n) const { return mul ? (int)__umulhi((unsigned)n, mul) : n; }
};

struct CcLevel {
  int n0, n1, n2;
  int hk;                             // pairs per row of the colour arrays: 2 ceil(n2 / 4)
  CcDiv by_qpl, by_hq, by_n0;         // quads of a plane, quads of a row, n0
  CcDiv by_crows, by_ck;              // (n1 / 2) (n2 / 2), n2 / 2
  short lo[CC_MAXC + 1];              // first plane of each slab (lo[A] = n0)
  int A, c0;                          // slabs of planes on CTAs c0 .. c0 + A - 1
  int smax;                           // planes of the largest slab
  int oP, oB;                         // float offsets: red and black p (halo planes included), the two right-hand-side slots
  const void* bx;
  const void* by;
  const void* bz;
};

struct CcArgs {
  int nl;  // levels swept here, [0] = top
  CcLevel L[PF_MG_MAX_LEVELS];
  int C;                // CTAs of the cluster
  int zero_floats;      // leading floats of shared memory that start at zero
  int oBar;             // four mbarriers: from the lower, upper neighbour, two in turn
  int oS;               // pair residuals of the level being restricted
  int oPd;              // FP64 p of a coarsest level swept in FP64 (even)
  int nb, bn1, bn2, cd; // dense level: cells, extents of axes 1 and 2, CTA holding its vectors (nb = 0: none)
  int oDB, oDP, oDb, oDr, oDM;  // its right-hand-side slots, solution; per CTA: b, partial sums, staged rows (-1: in L2)
  const void* M;        // M[m * nb + i], float (FP64 with 16-bit storage)
  const void* b;        // right-hand side of the top level
  int b_f32;            // b is float (else the storage type)
  const float* b_scale;
  void* p_out;
  float omega;
  int pre, post, coarsest;
  float rscale, pscale;
  int flux;
  MGState* st;
  int want_mean, mixed;
};

// ---- cluster primitives
__device__ __forceinline__ unsigned cc_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned cc_map(unsigned saddr, int rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cc_st(unsigned addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ void cc_st(unsigned addr, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}
// two floats to another CTA's shared memory, counted on that CTA's mbarrier
__device__ __forceinline__ void cc_st_async(unsigned addr, f2 v, unsigned bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(addr), "l"(v.v),
               "r"(bar)
               : "memory");
}
__device__ __forceinline__ bool cc_try_wait(unsigned bar, unsigned phase) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(phase)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ float cc_ld(unsigned addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ void cc_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cc_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ void cc_sync() {
  cc_arrive();
  cc_wait();
}

// slab r of A starts at plane r n0 / A; the slab that holds plane i
__device__ __forceinline__ int cc_owner(const CcLevel& L, int i) { return L.by_n0((i + 1) * L.A - 1); }

// the arithmetic type of the coarsest solve
template <class T> struct CcAcc { using type = double; };
template <> struct CcAcc<float> { using type = float; };

// four consecutive elements from a 4-element boundary, widened
__device__ __forceinline__ void cc_ld4(const float* p, float (&v)[4]) {
  const float4 q = __ldg(reinterpret_cast<const float4*>(p));
  v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
}
template <class T> __device__ __forceinline__ void cc_ld4(const T* p, float (&v)[4]) {
  union { uint2 u; T t[4]; } q;
  q.u = __ldg(reinterpret_cast<const uint2*>(p));
#pragma unroll
  for (int d = 0; d < 4; ++d) v[d] = ldT(q.t + d);
}

// this CTA's shared memory by 32-bit byte address
__device__ __forceinline__ f2 cc_lds2(unsigned addr) {
  f2 r;
  asm volatile("ld.shared.b64 %0, [%1];" : "=l"(r.v) : "r"(addr));
  return r;
}
__device__ __forceinline__ float cc_lds(unsigned addr) {
  float r;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(r) : "r"(addr));
  return r;
}
__device__ __forceinline__ double cc_ldsd(unsigned addr) {
  double r;
  asm volatile("ld.shared.f64 %0, [%1];" : "=d"(r) : "r"(addr));
  return r;
}
__device__ __forceinline__ void cc_sts2(unsigned addr, f2 v) {
  asm volatile("st.shared.b64 [%0], %1;" ::"r"(addr), "l"(v.v) : "memory");
}
__device__ __forceinline__ void cc_stsd(unsigned addr, double v) {
  asm volatile("st.shared.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}

// One CTA's share of the cycle.  Colour 0 ("red") is (i + j + k) even.
template <class T, int NQ> struct CoarseCycle {
  const CcArgs& a;
  float* sm;
  unsigned sm0;    // shared address of sm
  int tid, rank;
  int held;        // level whose coefficients are in the registers (-1: none)
  unsigned turn;   // halo exchanges so far, on any level
  unsigned phase;  // phase bits of the four mbarriers
  bool fail;       // a wait ran out: no more waits, the result is flagged
  unsigned bvec;   // shared address of the top level's right-hand side (0: a.b), and its scale
  float bvec_scale;
  // the level at hand
  int pl, cnt, s, lo, hk;
  unsigned P[2];      // shared addresses of the red and black arrays
  unsigned mlo, mhi;  // the neighbours' shared memory (0: none)
  int dlo;            // offset of the lower neighbour's upper halo against this CTA's first plane
  // quads: f2 holds the colour's cells of the quad's first and second pair
  f2 x0[2][NQ], x1[2][NQ], y0[2][NQ], y1[2][NQ], zo[2][NQ], zs[NQ], wd[2][NQ], b[2][NQ], p[2][NQ];
  unsigned par;       // bit u: parity of i + j of quad u

  __device__ __forceinline__ CoarseCycle(const CcArgs& a_, float* sm_) : a(a_), sm(sm_) {
    sm0 = smem_u32(sm_);
    tid = threadIdx.x;
    rank = (int)cc_rank();
    held = -1;
    turn = phase = par = 0u;
    fail = false;
    bvec = 0u;
    bvec_scale = 1.f;
  }

  __device__ __forceinline__ bool on(int u) const { return u * CC_NT + tid < cnt; }
  // index of quad u's first pair in the colour arrays
  __device__ __forceinline__ unsigned at(int u) const { return (unsigned)(pl + 2 * (u * CC_NT + tid)); }
  __device__ __forceinline__ int odd(int u) const { return (par >> u) & 1u; }

  __device__ __forceinline__ void init_barriers() {
    if (tid == 0) {
      for (int q = 0; q < 4; ++q)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sm0 + 4u * (unsigned)a.oBar + 8u * q) : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
  }

  // geometry of level l for this CTA
  __device__ __forceinline__ void enter(int l) {
    const CcLevel& L = a.L[l];
    const int r = rank - L.c0;
    const bool mine = r >= 0 && r < L.A;
    lo = mine ? L.lo[r] : 0;
    s = mine ? L.lo[r + 1] - lo : 0;
    hk = L.hk;
    pl = L.n1 * hk;
    cnt = s * (pl >> 1);
    P[0] = sm0 + 4u * (unsigned)L.oP;
    P[1] = P[0] + 4u * (unsigned)((L.smax + 2) * pl);
    mlo = mhi = 0u;
    dlo = 0;
    if (mine && r > 0) {
      mlo = cc_map(sm0, rank - 1);
      dlo = (lo - L.lo[r - 1]) * pl;
    }
    if (mine && r < L.A - 1) mhi = cc_map(sm0, rank + 1);
  }

  // row (li n1 + j) and quad within the row of quad u
  __device__ __forceinline__ void locate(const CcLevel& L, int u, int& row, int& h) const {
    const int e = u * CC_NT + tid;
    row = L.by_hq(e);
    h = e - row * (hk >> 1);
  }

  // face coefficients and omega/diagonal of the level's quads; a face on a wall
  // of the domain counts in the diagonal and has no neighbour
  __device__ __forceinline__ void load_coefs(int l) {
    if (held == l || s == 0) return;
    const CcLevel& L = a.L[l];
    load_faces(L, reinterpret_cast<const T*>(L.bx), reinterpret_cast<const T*>(L.by), reinterpret_cast<const T*>(L.bz));
    held = l;
  }

  template <class F> __device__ __forceinline__ void load_faces(const CcLevel& L, const F* X, const F* Y, const F* Z) {
    held = -1;
    par = 0u;
    const int n0 = L.n0, n1 = L.n1, n2 = L.n2;
    const bool wide = (n2 & 3) == 0 && ((reinterpret_cast<uintptr_t>(X) | reinterpret_cast<uintptr_t>(Y)) & 15u) == 0;
#pragma unroll
    for (int u = 0; u < NQ; ++u) {
      float xl[4], xu[4], yl[4], yu[4], z[5];
#pragma unroll
      for (int d = 0; d < 4; ++d) xl[d] = xu[d] = yl[d] = yu[d] = z[d] = 0.f;
      z[4] = 0.f;
      int i = 0, j = 0, h = 0;
      if (on(u)) {
        int row;
        locate(L, u, row, h);
        const int li = L.by_qpl(u * CC_NT + tid);
        j = row - li * n1;
        i = lo + li;
        const int r = i * n1 + j;
        const F* x = X + r * n2 + 4 * h;
        const F* y = Y + (r + i) * n2 + 4 * h;
        const F* zz = Z + r * (n2 + 1) + 4 * h;
        if (wide) {
          cc_ld4(x, xl);
          cc_ld4(x + n1 * n2, xu);
          cc_ld4(y, yl);
          cc_ld4(y + n2, yu);
        }
#pragma unroll
        for (int d = 0; d < 4; ++d) {
          if (4 * h + d >= n2) continue;
          if (!wide) {
            xl[d] = ldT(x + d);
            xu[d] = ldT(x + n1 * n2 + d);
            yl[d] = ldT(y + d);
            yu[d] = ldT(y + n2 + d);
          }
          z[d] = ldT(zz + d);
          z[d + 1] = ldT(zz + d + 1);
        }
      }
      const int o = (i + j) & 1;
      par |= (unsigned)o << u;
      float w[4];
#pragma unroll
      for (int d = 0; d < 4; ++d) {
        // cells past the row's end keep a zero diagonal
        const float dg = 4 * h + d < n2 ? xl[d] + xu[d] + yl[d] + yu[d] + z[d] + z[d + 1] : 0.f;
        w[d] = dg > 0.f ? a.omega / dg : 0.f;
        if (i == 0) xl[d] = 0.f;
        if (i == n0 - 1) xu[d] = 0.f;
        if (j == 0) yl[d] = 0.f;
        if (j == n1 - 1) yu[d] = 0.f;
      }
      if (h == 0) z[0] = 0.f;
#pragma unroll
      for (int d = 0; d < 4; ++d)
        if (4 * h + d >= n2 - 1) z[d + 1] = 0.f;
      // colour c holds cells d = o ^ c and 2 + (o ^ c); the face between a
      // pair's two cells is z[1] / z[3], the other one z[0], z[2] or z[2], z[4]
      zs[u] = f2_make(z[1], z[3]);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const bool hi = (o ^ c) != 0;
        x0[c][u] = hi ? f2_make(xl[1], xl[3]) : f2_make(xl[0], xl[2]);
        x1[c][u] = hi ? f2_make(xu[1], xu[3]) : f2_make(xu[0], xu[2]);
        y0[c][u] = hi ? f2_make(yl[1], yl[3]) : f2_make(yl[0], yl[2]);
        y1[c][u] = hi ? f2_make(yu[1], yu[3]) : f2_make(yu[0], yu[2]);
        wd[c][u] = hi ? f2_make(w[1], w[3]) : f2_make(w[0], w[2]);
        zo[c][u] = hi ? f2_make(z[2], z[4]) : f2_make(z[0], z[2]);
      }
    }
  }

  // the right-hand side of the level's quads: from global memory (top), or the
  // two plane sums the level above left in the slots
  __device__ __forceinline__ void load_b(int l) {
    if (l == 0 && bvec != 0u) {
      const f2 sc = f2_bcast(bvec_scale);
#pragma unroll
      for (int u = 0; u < NQ; ++u)
#pragma unroll
        for (int c = 0; c < 2; ++c) b[c][u] = f2_mul(vec(bvec, c, u), sc);
      return;
    }
    const CcLevel& L = a.L[l];
    const float bsc = l == 0 && a.b_scale ? *a.b_scale : 1.f;
    const size_t g0 = (size_t)lo * L.n1 * L.n2;
    const float* B = sm + L.oB;
    const int sl = L.smax * L.n1 * L.n2;
    const bool wide = (L.n2 & 3) == 0 && (l > 0 || (reinterpret_cast<uintptr_t>(a.b) & 15u) == 0);
    float v[NQ][4];
#pragma unroll
    for (int u = 0; u < NQ; ++u) {
#pragma unroll
      for (int d = 0; d < 4; ++d) v[u][d] = 0.f;
      if (!on(u)) continue;
      int row, h;
      locate(L, u, row, h);
      const int e = row * L.n2 + 4 * h;
      if (l == 0) {
        if (wide) {
          if (a.b_f32) cc_ld4(reinterpret_cast<const float*>(a.b) + g0 + e, v[u]);
          else cc_ld4(reinterpret_cast<const T*>(a.b) + g0 + e, v[u]);
        } else {
#pragma unroll
          for (int d = 0; d < 4; ++d)
            if (4 * h + d < L.n2)
              v[u][d] = a.b_f32 ? reinterpret_cast<const float*>(a.b)[g0 + e + d]
                                : ldT(reinterpret_cast<const T*>(a.b) + g0 + e + d);
        }
      } else {
#pragma unroll
        for (int d = 0; d < 4; ++d)
          if (4 * h + d < L.n2) v[u][d] = roundT<T>((B[e + d] + B[e + d + sl]) * a.rscale);
      }
    }
#pragma unroll
    for (int u = 0; u < NQ; ++u) {
      const bool o = odd(u);
      if (l == 0) {
#pragma unroll
        for (int d = 0; d < 4; ++d) v[u][d] *= bsc;
      }
      b[0][u] = o ? f2_make(v[u][1], v[u][3]) : f2_make(v[u][0], v[u][2]);
      b[1][u] = o ? f2_make(v[u][0], v[u][2]) : f2_make(v[u][1], v[u][3]);
    }
  }

  // a vector of the top level's cells private to their threads: f2 per colour and quad
  __device__ __forceinline__ unsigned vec_at(unsigned v, int c, int u) const {
    return v + 8u * (unsigned)((c * NQ + u) * CC_NT + tid);
  }
  __device__ __forceinline__ f2 vec(unsigned v, int c, int u) const { return cc_lds2(vec_at(v, c, u)); }

  // p of the level's quads from the shared arrays
  __device__ __forceinline__ void load_p() {
#pragma unroll
    for (int u = 0; u < NQ; ++u) {
      const f2 z = f2_bcast(0.f);
      p[0][u] = on(u) ? cc_lds2(P[0] + 4u * at(u)) : z;
      p[1][u] = on(u) ? cc_lds2(P[1] + 4u * at(u)) : z;
    }
  }

  // store the colour-C values of the quads; `halo`: in the neighbours' halo
  // planes too, as one exchange of `turn`.  Every step first computes all its
  // values, then stores them: its loads are in flight together.
  template <int C> __device__ __forceinline__ void put(const f2 (&v)[NQ], bool halo) {
#pragma unroll
    for (int u = 0; u < NQ; ++u) {
      p[C][u] = v[u];
      if (on(u)) cc_sts2(P[C] + 4u * at(u), v[u]);
    }
    if (!halo) return;
    if ((mlo | mhi) != 0u) {
      const unsigned off = P[C] - sm0;
      // the neighbour's barriers: [0, 1] data from below, [2, 3] from above
      const unsigned bar = 4u * (unsigned)a.oBar + 8u * (turn & 1u);
#pragma unroll
      for (int u = 0; u < NQ; ++u) {
        if (!on(u)) continue;
        const int q = (int)at(u);
        if (mlo != 0u && q < 2 * pl) cc_st_async(mlo + off + 4u * (unsigned)(q + dlo), v[u], mlo + bar + 16u);
        if (mhi != 0u && q >= s * pl) cc_st_async(mhi + off + 4u * (unsigned)(q - s * pl), v[u], mhi + bar);
      }
      if (tid == 0) {  // this CTA's share of the exchange
        const unsigned bytes = 4u * (unsigned)pl, own = sm0 + bar;
        if (mlo != 0u)
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(own), "r"(bytes) : "memory");
        if (mhi != 0u)
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(own + 16u), "r"(bytes) : "memory");
      }
    }
    ++turn;
  }

  __device__ __forceinline__ void wait_on(int q) {
    const unsigned bar = sm0 + 4u * (unsigned)a.oBar + 8u * (unsigned)q;
    const unsigned ph = (phase >> q) & 1u;
    unsigned it = 0;
    while (!fail && !cc_try_wait(bar, ph))
      if (++it > kTmaWaitLimit) fail = true;
    phase ^= 1u << q;
  }

  // end of a step on the level at hand after `n` exchanges: its CTAs see the
  // new values.  With a settle after every exchange, a neighbour's next store
  // into a halo plane cannot overtake this CTA's reads of it: it waits for the
  // stores of exactly the threads that read that plane.  Nor can its store after
  // next, on the same barrier and of the same colour, overtake this one: it
  // waits for this CTA's next exchange, which follows this settle.  Two
  // exchanges before one settle need a cluster barrier before the next exchange.
  __device__ __forceinline__ void settle(int n) {
    if (s == 0) return;
    __syncthreads();
    for (int q = n; q > 0; --q) {
      const int o = (int)((turn - (unsigned)q) & 1u);
      if (mlo != 0u) wait_on(o);
      if (mhi != 0u) wait_on(2 + o);
    }
  }

  // r[u] = b - A p at the colour-C cells: the row as the sum of beta (p - p_nbr)
  // (flux form), or as diag p - the sum of beta p_nbr
  template <int C> __device__ __forceinline__ void residual(f2 (&r)[NQ]) const {
    const unsigned dx = 4u * (unsigned)pl, dy = 4u * (unsigned)hk;
    const f2 m1 = f2_bcast(-1.f);
#pragma unroll
    for (int u = 0; u < NQ; ++u) {
      r[u] = f2_bcast(0.f);
      if (!on(u)) continue;
      const unsigned Q = P[1 - C] + 4u * at(u);
      const bool up = (odd(u) ^ C) != 0;  // the neighbours along k outside the pairs lie above
      const f2 pv = p[C][u], po = p[1 - C][u];
      const f2 qx0 = cc_lds2(Q - dx), qx1 = cc_lds2(Q + dx), qy0 = cc_lds2(Q - dy), qy1 = cc_lds2(Q + dy);
      const float qe = cc_lds(up ? Q + 8u : Q - 4u);
      const f2 qz = up ? f2_make(f2_y(po), qe) : f2_make(qe, f2_x(po));
      if (a.flux) {
        f2 t = f2_mul(x0[C][u], f2_fma(qx0, m1, pv));
        t = f2_fma(x1[C][u], f2_fma(qx1, m1, pv), t);
        t = f2_fma(y0[C][u], f2_fma(qy0, m1, pv), t);
        t = f2_fma(y1[C][u], f2_fma(qy1, m1, pv), t);
        t = f2_fma(zs[u], f2_fma(po, m1, pv), t);
        t = f2_fma(zo[C][u], f2_fma(qz, m1, pv), t);
        r[u] = f2_fma(t, m1, b[C][u]);
      } else {
        const f2 d = f2_add(f2_add(f2_add(f2_add(f2_add(x0[C][u], x1[C][u]), y0[C][u]), y1[C][u]), zs[u]), zo[C][u]);
        f2 t = f2_mul(x0[C][u], qx0);
        t = f2_fma(x1[C][u], qx1, t);
        t = f2_fma(y0[C][u], qy0, t);
        t = f2_fma(y1[C][u], qy1, t);
        t = f2_fma(zs[u], po, t);
        t = f2_fma(zo[C][u], qz, t);
        r[u] = f2_fma(f2_fma(t, m1, f2_mul(d, pv)), m1, b[C][u]);
      }
    }
  }

  template <int C> __device__ __forceinline__ void half_sweep(bool halo) {
    f2 v[NQ];
    residual<C>(v);
#pragma unroll
    for (int u = 0; u < NQ; ++u) v[u] = f2_fma(wd[C][u], v[u], p[C][u]);
    put<C>(v, halo);
    settle(halo ? 1 : 0);
  }

  // `last_halo`: whether anything reads the halos after the last half-sweep
  __device__ __forceinline__ void sweeps(int n, int reverse, bool last_halo) {
    for (int sw = 0; sw < 2 * n; ++sw) {
      const bool halo = last_halo || sw < 2 * n - 1;
      if (((sw & 1) ^ reverse) == 0) half_sweep<0>(halo);
      else half_sweep<1>(halo);
    }
  }

  // residual of the level summed over 1 x 2 x 2 cells of each plane, into the
  // slot (plane parity) of the next level's right-hand side at its owner
  __device__ __forceinline__ void restrict_to_next(int l) {
    const CcLevel& L = a.L[l];
    float* S = sm + a.oS;
    f2 r0[NQ], r1[NQ];
    residual<0>(r0);
    residual<1>(r1);
#pragma unroll
    for (int u = 0; u < NQ; ++u)
      if (on(u)) cc_sts2(smem_u32(S) + 4u * (at(u) - (unsigned)pl), f2_add(r0[u], r1[u]));
    __syncthreads();
    const int ck = L.n2 >> 1, rows = (L.n1 >> 1) * ck, m = s * rows;
    const bool swept = l + 1 < a.nl;
    if (!swept && L.A == 1) {  // this CTA has all of the dense level's right-hand side: to every CTA at once
      for (int e = tid; e < a.nb; e += CC_NT) {
        const int I = L.by_crows(e), t = e - I * rows, J = L.by_ck(t), k = t - J * ck;
        const int f = (2 * I * L.n1 + 2 * J) * hk + k;
        const float v = roundT<T>(((S[f] + S[f + hk]) + (S[f + pl] + S[f + pl + hk])) * a.rscale);
        for (int r = 0; r < a.C; ++r) cc_st(cc_map(sm0, r) + 4u * (unsigned)(a.oDb + e), v);
      }
      return;
    }
    const CcLevel& N = a.L[swept ? l + 1 : l];
    for (int e = tid; e < m; e += CC_NT) {
      const int li = L.by_crows(e), t = e - li * rows, J = L.by_ck(t), k = t - J * ck;
      const int f = (li * L.n1 + 2 * J) * hk + k;
      const int I = (lo + li) >> 1, slot = (lo + li) & 1;
      int cta = a.cd, off = a.oDB + slot * a.nb + I * rows + t;
      if (swept) {
        const int r = cc_owner(N, I);
        cta = N.c0 + r;
        off = N.oB + (slot * N.smax + I - N.lo[r]) * rows + t;
      }
      cc_st(cc_map(sm0, cta) + 4u * (unsigned)off, S[f] + S[f + hk]);
    }
  }

  // p += pscale * the coarse cell's p (one coarse cell per pair)
  __device__ __forceinline__ void prolong(int l) {
    const CcLevel& L = a.L[l];
    const bool swept = l + 1 < a.nl;
    const CcLevel& N = a.L[swept ? l + 1 : l];
    float va[NQ], vb[NQ];
#pragma unroll
    for (int u = 0; u < NQ; ++u) {
      va[u] = vb[u] = 0.f;
      if (!on(u)) continue;
      int row, h;
      locate(L, u, row, h);
      const int li = L.by_qpl(u * CC_NT + tid), j = row - li * L.n1, I = (lo + li) >> 1, J = j >> 1;
      if (swept) {  // coarse cells k = 2h and 2h + 1: one of each colour, both at pair h of their row
        const int r = cc_owner(N, I), pn = N.n1 * N.hk, sp = (N.smax + 2) * pn;
        const unsigned src = cc_map(sm0, N.c0 + r) + 4u * (unsigned)(N.oP + (I - N.lo[r] + 1) * pn + J * N.hk + h);
        const unsigned odd_row = (unsigned)((I + J) & 1) * 4u * (unsigned)sp;
        va[u] = cc_ld(src + odd_row);
        vb[u] = cc_ld(src + (4u * (unsigned)sp - odd_row));
      } else {
        const unsigned src = cc_map(sm0, a.cd) + 4u * (unsigned)(a.oDP + (I * a.bn1 + J) * a.bn2 + 2 * h);
        va[u] = cc_ld(src);
        if (2 * h + 1 < a.bn2) vb[u] = cc_ld(src + 4u);
      }
    }
    f2 v0[NQ], v1[NQ];
    const f2 sc = f2_bcast(a.pscale);
#pragma unroll
    for (int u = 0; u < NQ; ++u) {
      const f2 v = f2_make(va[u], vb[u]);
      v0[u] = f2_fma(v, sc, p[0][u]);
      v1[u] = f2_fma(v, sc, p[1][u]);
    }
    // one exchange, of colour 0: the post-sweeps begin with colour 1, which reads
    // colour 0 and then sends its own
    put<0>(v0, true);
    put<1>(v1, false);
    settle(1);
  }

  // sum over the CTAs of level l of a per-thread value, in every thread of them.
  // A CTA reads its s_part after the cluster barrier in here, so the next sum into
  // the same s_part needs another cluster barrier before it; sums without one take
  // another s_part.
  __device__ __forceinline__ double level_sum(int l, double v, double* sred, double* s_part) {
    const CcLevel& L = a.L[l];
    v = block_sum<CC_NT>(v, sred);
    if (L.A == 1) {
      if (tid == 0) s_part[0] = v;
      __syncthreads();
      return s_part[0];
    }
    if (tid == 0) s_part[CC_MAXC] = v;
    __syncthreads();
    if (s > 0 && tid < L.A) cc_st(cc_map(smem_u32(s_part + (rank - L.c0)), L.c0 + tid), s_part[CC_MAXC]);
    cc_sync();
    double t = 0.0;
    if (s > 0)
      for (int r = 0; r < L.A; ++r) t += s_part[r];
    return t;
  }

  // whether the quad's cells of colour c exist (a row may end inside its last
  // quad), and their FP32 diagonals
  __device__ __forceinline__ void present(const CcLevel& L, int u, int c, bool (&in)[2]) const {
    in[0] = in[1] = true;
    if ((L.n2 & 3) == 0) return;
    int row, h;
    locate(L, u, row, h);
    const int k = 4 * h + (odd(u) ^ c);
    in[0] = k < L.n2;
    in[1] = k + 2 < L.n2;
  }

  // p = round(v + shift) where the cell exists
  template <int C> __device__ __forceinline__ void put_shifted(const CcLevel& L, const double (&v)[2][NQ], double shift) {
    f2 w[NQ];
#pragma unroll
    for (int u = 0; u < NQ; ++u) {
      w[u] = p[C][u];  // a CTA outside this level still holds another level's p
      if (!on(u)) continue;
      bool in[2];
      present(L, u, C, in);
      w[u] = f2_make(in[0] ? roundT<T>((float)(v[0][u] + shift)) : 0.f, in[1] ? roundT<T>((float)(v[1][u] + shift)) : 0.f);
    }
    put<C>(w, false);
  }

  // FP64 sweeps of a coarsest level held by one CTA (16-bit hierarchy): pd[C] the
  // colour's values, wdd omega/diagonal
  template <int C>
  __device__ __forceinline__ void half_sweep_d(unsigned D0, unsigned D1, double (&pd)[2][2][NQ], const double (&wdd)[2][2][NQ]) {
#pragma unroll
    for (int u = 0; u < NQ; ++u) {
      if (!on(u)) continue;
      const bool up = (odd(u) ^ C) != 0;
      const float cx0[2] = {f2_x(x0[C][u]), f2_y(x0[C][u])}, cx1[2] = {f2_x(x1[C][u]), f2_y(x1[C][u])};
      const float cy0[2] = {f2_x(y0[C][u]), f2_y(y0[C][u])}, cy1[2] = {f2_x(y1[C][u]), f2_y(y1[C][u])};
      const float czs[2] = {f2_x(zs[u]), f2_y(zs[u])}, czo[2] = {f2_x(zo[C][u]), f2_y(zo[C][u])};
      const float cb[2] = {f2_x(b[C][u]), f2_y(b[C][u])};
      const unsigned Q = (C ? D0 : D1) + 8u * at(u), dx = 8u * (unsigned)pl, dy = 8u * (unsigned)hk;
      const double qe = cc_ldsd(up ? Q + 16u : Q - 8u);
      double v[2];
#pragma unroll
      for (int d = 0; d < 2; ++d) {
        const double pv = pd[C][d][u], po = pd[1 - C][d][u];
        const double qz = up == (d == 1) ? qe : pd[1 - C][1 - d][u];
        double res;
        if (a.flux) {
          double t = (double)cx0[d] * (pv - cc_ldsd(Q + 8u * d - dx));
          t += (double)cx1[d] * (pv - cc_ldsd(Q + 8u * d + dx));
          t += (double)cy0[d] * (pv - cc_ldsd(Q + 8u * d - dy));
          t += (double)cy1[d] * (pv - cc_ldsd(Q + 8u * d + dy));
          t += (double)czs[d] * (pv - po);
          t += (double)czo[d] * (pv - qz);
          res = (double)cb[d] - t;
        } else {
          const double dg = (double)(cx0[d] + cx1[d] + cy0[d] + cy1[d] + czs[d] + czo[d]);
          double t = (double)cx0[d] * cc_ldsd(Q + 8u * d - dx);
          t += (double)cx1[d] * cc_ldsd(Q + 8u * d + dx);
          t += (double)cy0[d] * cc_ldsd(Q + 8u * d - dy);
          t += (double)cy1[d] * cc_ldsd(Q + 8u * d + dy);
          t += (double)czs[d] * po;
          t += (double)czo[d] * qz;
          res = (double)cb[d] - (dg * pv - t);
        }
        v[d] = pv + res * wdd[C][d][u];
      }
      const unsigned W = (C ? D1 : D0) + 8u * at(u);
#pragma unroll
      for (int d = 0; d < 2; ++d) {
        pd[C][d][u] = v[d];
        cc_stsd(W + 8u * d, v[d]);
      }
    }
  }

  // `coarsest` sweeps from zero and the mean removed (pfflip/poisson.py:325-328)
  __device__ __forceinline__ void coarsest_solve(int l, double* sred, double* s_part) {
    const CcLevel& L = a.L[l];
    const double n = (double)L.n0 * L.n1 * L.n2;
    constexpr bool kF64 = !std::is_same<T, float>::value;
    if constexpr (kF64) {
      if (L.A == 1) {
        if (s == 0) return;
        const unsigned D0 = sm0 + 4u * (unsigned)a.oPd, D1 = D0 + 8u * (unsigned)((s + 2) * pl);
        double pd[2][2][NQ], wdd[2][2][NQ];
#pragma unroll
        for (int u = 0; u < NQ; ++u) {
          int row = 0, h = 0;
          if (on(u)) locate(L, u, row, h);
          const int li = L.by_qpl(on(u) ? u * CC_NT + tid : 0), j = row - li * L.n1, r = (lo + li) * L.n1 + j;
#pragma unroll
          for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int d = 0; d < 2; ++d) {
              pd[c][d][u] = 0.0;
              const int k = 4 * h + 2 * d + (odd(u) ^ c);
              float dg = 0.f;
              if (on(u) && k < L.n2) {
                const T* X = reinterpret_cast<const T*>(L.bx) + r * L.n2 + k;
                const T* Y = reinterpret_cast<const T*>(L.by) + (r + lo + li) * L.n2 + k;
                const T* Z = reinterpret_cast<const T*>(L.bz) + r * (L.n2 + 1) + k;
                dg = ldT(X) + ldT(X + L.n1 * L.n2) + ldT(Y) + ldT(Y + L.n2) + ldT(Z) + ldT(Z + 1);
              }
              wdd[c][d][u] = dg > 0.f ? (double)a.omega / (double)dg : 0.0;
            }
        }
        for (int sw = 0; sw < a.coarsest; ++sw) {
          half_sweep_d<0>(D0, D1, pd, wdd);
          __syncthreads();
          half_sweep_d<1>(D0, D1, pd, wdd);
          __syncthreads();
        }
        double t = 0.0;
#pragma unroll
        for (int u = 0; u < NQ; ++u)
#pragma unroll
          for (int d = 0; d < 2; ++d) t += pd[0][d][u] + pd[1][d][u];
        const double shift = -level_sum(l, t, sred, s_part) / n;
        put_shifted<0>(L, pd[0], shift);
        put_shifted<1>(L, pd[1], shift);
        return;
      }
    }
    sweeps(a.coarsest, 0, false);
    double v[2][2][NQ], t = 0.0;
#pragma unroll
    for (int u = 0; u < NQ; ++u)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        v[c][0][u] = (double)f2_x(p[c][u]);
        v[c][1][u] = (double)f2_y(p[c][u]);
        if (on(u)) t += v[c][0][u] + v[c][1][u];
      }
    const double mean = level_sum(l, t, sred, s_part) / n;
    put_shifted<0>(L, v[0], (double)(float)(-mean));
    put_shifted<1>(L, v[1], (double)(float)(-mean));
  }

  // ---- the dense operator: CTA r applies rows [r R, (r + 1) R), R = ceil(nb / C);
  // thread (i, c) the column chunk c of row i
  __device__ __forceinline__ void stage_dense() {
    if (a.nb == 0 || a.oDM < 0) return;
    using Acc = typename CcAcc<T>::type;
    const int R = (a.nb + a.C - 1) / a.C, row0 = rank * R, nr = min(R, a.nb - row0);
    if (nr <= 0) return;
    const int ch = CC_NT / R, c = tid / R, i = tid - c * R;
    if (c >= ch || i >= nr) return;
    const Acc* M = reinterpret_cast<const Acc*>(a.M) + row0 + i;
    Acc* D = reinterpret_cast<Acc*>(sm + a.oDM) + i;
    for (int m = c; m < a.nb; m += ch) {
      const unsigned dst = smem_u32(D + m * R);
      if (sizeof(Acc) == 8)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(M + (size_t)m * a.nb) : "memory");
      else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(M + (size_t)m * a.nb) : "memory");
    }
  }

  __device__ __forceinline__ void dense_solve() {
    using Acc = typename CcAcc<T>::type;
    const int nb = a.nb, R = (nb + a.C - 1) / a.C, row0 = rank * R, nr = min(R, nb - row0);
    float* bv = sm + a.oDb;
    Acc* red = reinterpret_cast<Acc*>(sm + a.oDr);
    if (nr > 0 && a.L[a.nl - 1].A > 1) {  // otherwise the level above has sent it
      const unsigned src = cc_map(sm0, a.cd) + 4u * (unsigned)a.oDB;
      for (int m = tid; m < nb; m += CC_NT)
        bv[m] = roundT<T>((cc_ld(src + 4u * (unsigned)m) + cc_ld(src + 4u * (unsigned)(m + nb))) * a.rscale);
    }
    __syncthreads();
    if (nr <= 0) return;
    const int ch = CC_NT / R, cw = (nb + ch - 1) / ch;
    const int c = tid / R, i = tid - c * R;
    if (c < ch && i < nr) {
      const int m0 = c * cw, m1 = min(nb, m0 + cw);
      Acc acc = Acc(0);
      if (a.oDM >= 0) {
        const Acc* D = reinterpret_cast<const Acc*>(sm + a.oDM) + i;
#pragma unroll 4
        for (int m = m0; m < m1; ++m) acc = fma(D[m * R], (Acc)bv[m], acc);
      } else {
        const Acc* M = reinterpret_cast<const Acc*>(a.M) + row0 + i;
#pragma unroll 8
        for (int m = m0; m < m1; ++m) acc = fma(__ldg(M + (size_t)m * nb), (Acc)bv[m], acc);
      }
      red[c * R + i] = acc;
    }
    __syncthreads();
    const unsigned dst = cc_map(sm0, a.cd) + 4u * (unsigned)(a.oDP + row0);
    for (int q = tid; q < nr; q += CC_NT) {
      Acc v = Acc(0);
      for (int t = 0; t < ch; ++t) v += red[t * R + q];
      cc_st(dst + 4u * (unsigned)q, roundT<T>((float)v));
    }
  }

  // one V-cycle from zero with the top level's right-hand side (already in the
  // registers); the top level's p is in the registers of its CTAs at the end
  __device__ __forceinline__ void cycle(double* sred, double* s_part) {
    const int nd = a.nb > 0 ? a.nl : a.nl - 1;  // levels smoothed on the way down
    for (int l = 0; l < a.nl; ++l) {
      enter(l);
      load_coefs(l);
      if (s > 0) {
        if (l > 0) load_b(l);
#pragma unroll
        for (int u = 0; u < NQ; ++u) p[0][u] = p[1][u] = f2_bcast(0.f);
      }
      if (l >= nd) break;
      sweeps(a.pre, 0, true);
      if (s > 0) restrict_to_next(l);
      cc_sync();
    }
    if (a.nb > 0) dense_solve();
    else coarsest_solve(a.nl - 1, sred, s_part);
    int at_hand = a.nl - 1;
    for (int l = nd - 1; l >= 0; --l) {
      cc_sync();  // the coarse solution is complete
      if (l != at_hand) {
        enter(l);
        at_hand = l;
        if (s > 0 && held != l) {  // another level's sweeps took the registers
          load_coefs(l);
          load_b(l);
          load_p();
        }
      }
      if (s > 0) prolong(l);
      else ++turn;
      if (l == 0) cc_arrive();  // done with the other CTAs' shared memory
      sweeps(a.post, 1, false);
    }
    // a CTA may leave, or start over, only when no other reads its shared memory
    if (nd > 0) cc_wait();
  }
};

template <class T, int NQ>
__global__ void __launch_bounds__(CC_NT, 1) k_coarse(const __grid_constant__ CcArgs a) {
  extern __shared__ __align__(16) float ccsm[];
  __shared__ double sred[40];
  __shared__ double s_part[CC_MAXC + 1], s_mean[CC_MAXC + 1];
  CoarseCycle<T, NQ> cy(a, ccsm);
  cy.stage_dense();
  cy.init_barriers();
  for (int l = 0; l < a.nl; ++l) {  // the first level this CTA has a part in
    cy.enter(l);
    if (cy.s > 0) {
      cy.load_coefs(l);
      break;
    }
  }
  for (int e = cy.tid; e < a.zero_floats / 4; e += CC_NT) reinterpret_cast<float4*>(ccsm)[e] = make_float4(0.f, 0.f, 0.f, 0.f);
  asm volatile("cp.async.wait_all;" ::: "memory");
  grid_dep_wait();
  if (is_done(a.st)) return;  // the same for every CTA; nothing remote has been touched
  cy.enter(0);
  if (cy.s > 0) cy.load_b(0);
  cc_sync();
  cy.cycle(sred, s_part);
  cy.enter(0);
  const CcLevel& L = a.L[0];
  T* out = reinterpret_cast<T*>(a.p_out) + (size_t)cy.lo * L.n1 * L.n2;
  double ls = 0.0;
#pragma unroll
  for (int u = 0; u < NQ; ++u) {
    if (!cy.on(u)) continue;
    int row, h;
    cy.locate(L, u, row, h);
    const f2 e0 = cy.odd(u) ? cy.p[1][u] : cy.p[0][u], e1 = cy.odd(u) ? cy.p[0][u] : cy.p[1][u];
    const float v[4] = {f2_x(e0), f2_x(e1), f2_y(e0), f2_y(e1)};
#pragma unroll
    for (int d = 0; d < 4; ++d) {
      if (4 * h + d >= L.n2) continue;
      stT(out + row * L.n2 + 4 * h + d, v[d]);
      ls += (double)roundT<T>(v[d]);
    }
  }
  if (a.want_mean) {
    const double tot = cy.level_sum(0, ls, sred, s_mean);
    if (cy.rank == L.c0 && cy.tid == 0) {
      const double n = (double)L.n0 * L.n1 * L.n2;
      a.st->sum_last = tot;
      a.st->c_shift = (float)(-(tot / n) * (a.mixed ? (double)a.st->zscale : 1.0));
    }
  }
  if (cy.fail && a.st) {
    a.st->status = ST_TMA_TIMEOUT;
    a.st->done = 1;
  }
}

// ---------------------------------------------------------------- the whole solve in the cluster
// Where k_coarse covers every level, the flexible CG around it runs in the same
// launch: r, x and A q stay in shared memory private to the threads that own
// the cells, q in two colour arrays with halo planes like p, the scalars in
// every thread.  An iteration is then the V-cycle and three reductions (q A q,
// max|r|, and the mean of z together with the dot products, since
// <r, z + c> = <r, z> + c <r, 1>) instead of six launches and a copy back.
// Sums are FP64 per thread, combined in a fixed order; the update formulas are
// those of the launched path (pfflip/poisson.py:355-409).
//
// Bound by the same chains as k_coarse, plus about 1 us a reduction.  Measured on
// a B200 against the launched CG around k_coarse, us: 32^3 solve to 1e-4 829 ->
// 555, four 16^3 steps 2924 -> 1938, a 24^3 gradient of two steps 6700 -> 4664.
constexpr int CC_RED = 4;  // values reduced at once

struct CcSolveArgs {
  CcArgs cc;
  float* x;        // solution, mean removed
  float* x_raw;    // what the launched CG leaves in its vectors: x before that,
  float* rhs;      // b without its mean (may be null),
  float* res[2];   // and the last two residuals, in turn
  float tol;
  int max_iter;
  float coef_scale;
  const float* bx;  // FP32 faces of the top level: the CG's operator
  const float* by;
  const float* bz;
  int n_total;
  int oQ;          // q: colour arrays with halos, as level 0's p
  int oR, oR2, oX; // vectors of f2 (16-byte aligned)
};

template <class T, int NQ>
__global__ void __launch_bounds__(CC_NT, 1) k_solve(const __grid_constant__ CcSolveArgs A) {
  extern __shared__ __align__(16) float ccsm[];
  __shared__ double sred[40];
  __shared__ double s_part[CC_MAXC + 1];
  __shared__ double s_warp[CC_RED][CC_NT / 32];
  __shared__ double s_all[2][CC_RED][CC_MAXC];
  __shared__ int s_go[2];
  __shared__ int s_fail;  // in the top level's first CTA: a wait of some thread of the cluster ran out
  const CcArgs& a = A.cc;
  CoarseCycle<T, NQ> cy(a, ccsm);
  const int tid = cy.tid;
  if (tid == 0) s_fail = 0;
  const CcLevel& L = a.L[0];
  cy.stage_dense();
  cy.init_barriers();
  for (int l = 0; l < a.nl; ++l) {
    cy.enter(l);
    if (cy.s > 0) {
      cy.load_coefs(l);
      break;
    }
  }
  const int nq4 = (L.smax + 2) * L.n1 * L.hk / 2;  // q: 2 (smax + 2) n1 hk floats
  auto rezero = [&]() {
    for (int e = tid; e < a.zero_floats / 4; e += CC_NT)
      reinterpret_cast<float4*>(ccsm)[e] = make_float4(0.f, 0.f, 0.f, 0.f);
  };
  rezero();
  for (int e = tid; e < nq4; e += CC_NT) reinterpret_cast<float4*>(ccsm + A.oQ)[e] = make_float4(0.f, 0.f, 0.f, 0.f);
  asm volatile("cp.async.wait_all;" ::: "memory");

  // sums (MAX: maxima) of K per-thread values over the top level's CTAs, in
  // every thread that needs them: those CTAs (A == 1), or all of the cluster
  unsigned red_turn = 0;
  auto reduce = [&](auto kc, auto is_max, double (&v)[CC_RED]) {
    constexpr int K = decltype(kc)::value;
    constexpr bool MAX = decltype(is_max)::value;
    const int lane = tid & 31, w = tid >> 5;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      double t = v[k];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const double q = __shfl_xor_sync(0xffffffffu, t, o);
        t = MAX ? fmax(t, q) : t + q;
      }
      if (lane == 0) s_warp[k][w] = t;
    }
    __syncthreads();
    const unsigned buf = red_turn++ & 1u;
    if (w < K) {
      double t = lane < CC_NT / 32 ? s_warp[w][lane] : 0.0;
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) {
        const double q = __shfl_xor_sync(0xffffffffu, t, o);
        t = MAX ? fmax(t, q) : t + q;
      }
      if (L.A == 1) {
        if (lane == 0) s_all[buf][w][0] = t;
      } else if (cy.s > 0 && lane < a.C) {
        cc_st(cc_map(smem_u32(&s_all[buf][w][cy.rank - L.c0]), lane), t);
      }
    }
    if (L.A == 1) __syncthreads();
    else cc_sync();
#pragma unroll
    for (int k = 0; k < K; ++k) {
      double t = s_all[buf][k][0];
      for (int r = 1; r < L.A; ++r) t = MAX ? fmax(t, s_all[buf][k][r]) : t + s_all[buf][k][r];
      v[k] = t;
    }
  };
  auto k1 = std::integral_constant<int, 1>();
  auto k4 = std::integral_constant<int, 4>();
  auto sum = std::false_type();
  auto mx = std::true_type();
  // the decision of the top level's CTAs, known to the cluster
  unsigned go_turn = 0;
  auto agree = [&](bool go) {
    if (L.A > 1 || a.C == 1) return go;
    const unsigned buf = go_turn++ & 1u;
    if (cy.s > 0 && tid < a.C) {
      unsigned at = cc_map(smem_u32(&s_go[buf]), tid);
      asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(at), "r"(go ? 1 : 0) : "memory");
    }
    cc_sync();
    return s_go[buf] != 0;
  };

  if (a.C > 1) cc_sync();
  else __syncthreads();
  cy.enter(0);
  const bool mine = cy.s > 0;
  const unsigned sm0 = cy.sm0, Rv[2] = {sm0 + 4u * (unsigned)A.oR, sm0 + 4u * (unsigned)A.oR2};
  const unsigned Xv = sm0 + 4u * (unsigned)A.oX;
  int cur = 0;
  unsigned in = 0u;  // bit 4 u + 2 c + d: cell d of colour c of quad u exists
  double red[CC_RED];

  // ---- r = b - mean(b), x = 0, |b|   (pfflip/poisson.py:363-372)
  red[0] = 0.0;
  if (mine) {
    cy.load_b(0);
#pragma unroll
    for (int u = 0; u < NQ; ++u)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        bool e[2] = {false, false};
        if (cy.on(u)) cy.present(L, u, c, e);
        in |= (e[0] ? 1u : 0u) << (4 * u + 2 * c) | (e[1] ? 2u : 0u) << (4 * u + 2 * c);
        red[0] += (double)f2_x(cy.b[c][u]) + (double)f2_y(cy.b[c][u]);
      }
  }
  auto masked = [&](int c, int u, float x, float y) {
    const unsigned m = in >> (4 * u + 2 * c);
    return f2_make(m & 1u ? x : 0.f, m & 2u ? y : 0.f);
  };
  // a vector of the top level's cells plus a constant, to global memory
  auto store = [&](float* g, unsigned v, float shift) {
    float* out = g + (size_t)cy.lo * L.n1 * L.n2;
#pragma unroll
    for (int u = 0; u < NQ; ++u) {
      if (!mine || !cy.on(u)) continue;
      int row, h;
      cy.locate(L, u, row, h);
      const f2 e0 = cy.vec(v, cy.odd(u), u), e1 = cy.vec(v, 1 - cy.odd(u), u);
      const float w[4] = {f2_x(e0), f2_x(e1), f2_y(e0), f2_y(e1)};
#pragma unroll
      for (int d = 0; d < 4; ++d)
        if (4 * h + d < L.n2) out[row * L.n2 + 4 * h + d] = w[d] + shift;
    }
  };
  auto amax = [](float x, float m) { return fmaxf(m, isfinite(x) ? fabsf(x) : INFINITY); };
  reduce(k1, sum, red);
  const double n = (double)A.n_total;
  float m = 0.f;
  {
    const float c0 = (float)(-(red[0] / n));
#pragma unroll
    for (int u = 0; u < NQ; ++u)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        if (!mine || !cy.on(u)) continue;
        const f2 r = masked(c, u, f2_x(cy.b[c][u]) + c0, f2_y(cy.b[c][u]) + c0);
        m = amax(f2_x(r), m);
        m = amax(f2_y(r), m);
        cc_sts2(cy.vec_at(Rv[0], c, u), r);
        cc_sts2(cy.vec_at(Xv, c, u), f2_bcast(0.f));
      }
  }
  if (A.rhs) store(A.rhs, Rv[0], 0.f);
  red[0] = (double)m;
  reduce(k1, mx, red);
  const double bnorm = red[0];
  double rel = 1.0, rz = 0.0, sum_r_old = 0.0;
  int it = 0, updates = 0, status = ST_RUNNING;
  bool go = A.max_iter > 0;
  if (!(bnorm > 0.0) || isinf(bnorm)) {
    status = bnorm == 0.0 ? ST_ZERO_RHS : ST_NONFINITE;
    rel = bnorm == 0.0 ? 0.0 : 1.0;
    go = false;
  }
  // 16-bit hierarchy: the top right-hand side is r * scale_r, a power of two
  // putting max|r| in [0.5, 1)
  float scale_r = 1.f;
  auto rescale = [&](double mr) {
    int ex = 0;
    frexpf(mr > 0.0 ? (float)mr : 1.f, &ex);
    if (a.mixed) scale_r = ldexpf(1.f, -ex);
  };
  rescale(bnorm);
  bool first = true;
  while (agree(go)) {
    // ---- z = V-cycle(r) with its mean removed
    cy.bvec = Rv[cur];
    cy.bvec_scale = scale_r;
    cy.enter(0);
    if (mine) {
      cy.load_coefs(0);
      cy.load_b(0);
    }
    cy.cycle(sred, s_part);
    __syncthreads();
    rezero();  // for the next cycle; a reduction or a cluster barrier comes first
    cy.enter(0);
    const float zs = a.mixed ? A.coef_scale / scale_r : 1.f;
#pragma unroll
    for (int k = 0; k < CC_RED; ++k) red[k] = 0.0;
#pragma unroll
    for (int u = 0; u < NQ; ++u)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        if (!mine || !cy.on(u)) continue;
        const f2 p = masked(c, u, roundT<T>(f2_x(cy.p[c][u])) * zs, roundT<T>(f2_y(cy.p[c][u])) * zs);
        const f2 rn = cy.vec(Rv[cur], c, u), ro = cy.vec(Rv[cur ^ 1], c, u);
        cy.p[c][u] = p;
        const double px = f2_x(p), py = f2_y(p);
        red[0] += px + py;
        red[1] += (double)f2_x(rn) * px + (double)f2_y(rn) * py;
        if (!first) red[2] += (double)f2_x(ro) * px + (double)f2_y(ro) * py;
        red[3] += (double)f2_x(rn) + (double)f2_y(rn);
      }
    reduce(k4, sum, red);
    const float cs = (float)(-(red[0] / n));
    const double rz_new = red[1] + (double)cs * red[3], rpz = red[2] + (double)cs * sum_r_old;
    const float beta = first || rz == 0.0 ? 0.f : (float)fmax((rz_new - rpz) / rz, 0.0);
    rz = rz_new;
    sum_r_old = red[3];
    // ---- q = z + beta q, A q, <q, A q>
    cy.P[0] = sm0 + 4u * (unsigned)A.oQ;
    cy.P[1] = cy.P[0] + 4u * (unsigned)((L.smax + 2) * cy.pl);
    red[0] = 0.0;
    if (mine) {
      f2 q0[NQ], q1[NQ];
#pragma unroll
      for (int u = 0; u < NQ; ++u) {
        q0[u] = q1[u] = f2_bcast(0.f);
        if (!cy.on(u)) continue;
        const f2 o0 = cc_lds2(cy.P[0] + 4u * cy.at(u)), o1 = cc_lds2(cy.P[1] + 4u * cy.at(u));
        q0[u] = masked(0, u, (f2_x(cy.p[0][u]) + cs) + beta * f2_x(o0), (f2_y(cy.p[0][u]) + cs) + beta * f2_y(o0));
        q1[u] = masked(1, u, (f2_x(cy.p[1][u]) + cs) + beta * f2_x(o1), (f2_y(cy.p[1][u]) + cs) + beta * f2_y(o1));
        cy.b[0][u] = cy.b[1][u] = f2_bcast(0.f);
      }
      cy.template put<0>(q0, true);
      cy.template put<1>(q1, true);
      // the 16-bit coefficients give way to the FP32 ones for this product
      if (!std::is_same<T, float>::value) cy.load_faces(L, A.bx, A.by, A.bz);
      cy.settle(2);
      cy.template residual<0>(q0);  // - A q
      cy.template residual<1>(q1);
#pragma unroll
      for (int u = 0; u < NQ; ++u) {
        if (!cy.on(u)) continue;
        red[0] -= (double)f2_x(cy.p[0][u]) * (double)f2_x(q0[u]) + (double)f2_y(cy.p[0][u]) * (double)f2_y(q0[u]);
        red[0] -= (double)f2_x(cy.p[1][u]) * (double)f2_x(q1[u]) + (double)f2_y(cy.p[1][u]) * (double)f2_y(q1[u]);
        // the older residual is used up: its place takes - A q, then the new one
        cc_sts2(cy.vec_at(Rv[cur ^ 1], 0, u), q0[u]);
        cc_sts2(cy.vec_at(Rv[cur ^ 1], 1, u), q1[u]);
      }
    } else {
      cy.turn += 2u;
    }
    reduce(k1, sum, red);
    const double qAq = red[0];
    ++it;
    first = false;
    if (!(qAq > 0.0)) {
      status = qAq <= 0.0 ? ST_BREAKDOWN : ST_NONFINITE;
      go = false;
    }
    // ---- x += alpha q, r -= alpha A q, |r|   (pfflip/poisson.py:390-398)
    const float al = go ? (float)(rz / qAq) : 0.f;
    m = 0.f;
    if (go) {
#pragma unroll
      for (int u = 0; u < NQ; ++u)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          if (!mine || !cy.on(u)) continue;
          const f2 x = cy.vec(Xv, c, u), r = cy.vec(Rv[cur], c, u), Aq = cy.vec(Rv[cur ^ 1], c, u), af = f2_bcast(al);
          const f2 rn = f2_fma(af, Aq, r);
          m = amax(f2_x(rn), m);
          m = amax(f2_y(rn), m);
          cc_sts2(cy.vec_at(Xv, c, u), f2_fma(af, cy.p[c][u], x));
          cc_sts2(cy.vec_at(Rv[cur ^ 1], c, u), rn);
        }
      cur ^= 1;
      ++updates;
    }
    red[0] = cy.fail ? (double)INFINITY : (double)m;  // a wait that ran out ends the iteration everywhere
    reduce(k1, mx, red);
    if (go) {
      rel = red[0] / bnorm;
      if (!(rel == rel) || isinf(rel)) {
        status = ST_NONFINITE;
        go = false;
      } else if (rel < (double)A.tol) {
        status = ST_CONVERGED;
        go = false;
      }
      if (it >= A.max_iter) go = false;
      rescale(red[0]);
    }
  }

  store(A.res[updates & 1], Rv[cur], 0.f);
  if (updates > 0 && updates == it) store(A.res[(updates & 1) ^ 1], Rv[cur ^ 1], 0.f);
  store(A.x_raw, Xv, 0.f);

  // ---- x with its mean removed
  red[0] = 0.0;
#pragma unroll
  for (int u = 0; u < NQ; ++u)
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      if (!mine || !cy.on(u)) continue;
      const f2 x = cy.vec(Xv, c, u);
      red[0] += (double)f2_x(x) + (double)f2_y(x);
    }
  reduce(k1, sum, red);
  store(A.x, Xv, (float)(-(red[0] / n)));
  if (cy.fail)
    asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(cc_map(smem_u32(&s_fail), L.c0)), "r"(1) : "memory");
  if (a.C > 1) cc_sync();  // no CTA leaves while another may still write to it
  else __syncthreads();
  if (cy.rank == L.c0 && tid == 0) {
    a.st->it = it;
    a.st->rel = rel;
    a.st->bnorm = bnorm;
    a.st->status = s_fail ? ST_TMA_TIMEOUT : status;
    a.st->done = 1;
  }
}

}  // namespace pf
