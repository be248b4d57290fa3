// Device code of the classic tile body that the interpreted kernels
// (tile_kernels_impl.cuh) and the FP64 passes compiled at run time (jit.cu)
// share: the ops on a thread's 16 amplitudes, the reduced matrices of the
// reverse sweep, and a pass's prologue, stage loads and stores, and epilogue.
// No host headers (the run-time compiler reads it too).
#pragma once

#include "cplx.cuh"
#include "tile_dev.cuh"

namespace vqc {

// ----------------------------------------------------------------------------- one-qubit ops
// Products with every rounding written out, so that the interpreted and the
// compiled form of a pass give the same bits.
template <class C>
__device__ __forceinline__ C tmul(C a, C b) {
  C r;
  r.x = fma(a.x, b.x, -a.y * b.y);
  r.y = fma(a.y, b.x, a.x * b.y);
  return r;
}
template <class C>
__device__ __forceinline__ C tfma(C a, C b, C acc) {
  acc.x = fma(a.x, b.x, acc.x);
  acc.x = fma(-a.y, b.y, acc.x);
  acc.y = fma(a.x, b.y, acc.y);
  acc.y = fma(a.y, b.x, acc.y);
  return acc;
}

// U on one pair.  The structured forms round like the general one (a product
// with an exact zero left out), so that a gate's bits do not depend on its form.
template <int FORM, class C>
__device__ __forceinline__ void u1_apply(C& x0, C& x1, const C (&u)[4]) {
  const C a = x0, b = x1;
  if (FORM == kFormGen) {
    x0 = tfma(u[1], b, tmul(u[0], a));
    x1 = tfma(u[3], b, tmul(u[2], a));
  } else if (FORM == kFormRI) {  // u00 = p, u01 = i q, u10 = i r, u11 = s (p, q, r, s real)
    x0.x = fma(-u[1].y, b.y, u[0].x * a.x);
    x0.y = fma(u[1].y, b.x, u[0].x * a.y);
    x1.x = fma(u[3].x, b.x, -u[2].y * a.y);
    x1.y = fma(u[3].x, b.y, u[2].y * a.x);
  } else if (FORM == kFormReal) {
    x0.x = fma(u[1].x, b.x, u[0].x * a.x);
    x0.y = fma(u[1].x, b.y, u[0].x * a.y);
    x1.x = fma(u[3].x, b.x, u[2].x * a.x);
    x1.y = fma(u[3].x, b.y, u[2].x * a.y);
  } else if (FORM == kFormDiag) {
    x0 = tmul(u[0], a);
    x1.x = fma(-u[3].y, b.y, u[3].x * b.x);
    x1.y = fma(u[3].y, b.x, u[3].x * b.y);
  } else if (FORM == kFormUD) {
    x0 = tfma(u[1], b, a);
    x1 = tfma(u[2], a, b);
  } else if (FORM == kFormRC) {
    const C t0 = tmul(u[1], b), t1 = tmul(u[2], a);
    x0.x = fma(u[0].x, a.x, t0.x);
    x0.y = fma(u[0].x, a.y, t0.y);
    x1.x = fma(u[3].x, b.x, t1.x);
    x1.y = fma(u[3].x, b.y, t1.y);
  } else if (FORM == kFormOff) {
    x0 = tmul(u[1], b);
    x1 = tmul(u[2], a);
  } else if (FORM == kFormSwap) {
    x0 = b;
    x1 = a;
  }
}

// Pair p of register slot RR: amplitudes j0 (target bit clear) and j0 | 1 << RR.
template <int RR>
__device__ __forceinline__ constexpr int pair_lo(int p) {
  return ((p >> RR) << (RR + 1)) | (p & ((1 << RR) - 1));
}

// MASK: pair p runs when bit j0 of rm is set (uniform over the grid).
template <int RR, bool MASK, int FORM, bool ADJ, class C>
__device__ __forceinline__ void op_u1(C (&v)[16], C (&w)[16], const C* U, uint32_t rm) {
  const C u[4] = {U[0], U[1], U[2], U[3]};
#pragma unroll
  for (int p = 0; p < 8; ++p) {
    const int j0 = pair_lo<RR>(p), j1 = j0 | (1 << RR);
    if (MASK && !((rm >> j0) & 1)) continue;
    u1_apply<FORM>(v[j0], v[j1], u);
    if (ADJ) u1_apply<FORM>(w[j0], w[j1], u);
  }
}

// ----------------------------------------------------------------------------- two-qubit and diagonal ops
template <class C>
__device__ __forceinline__ void u2_quad(C& x0, C& x1, C& x2, C& x3, const C* U) {
  const C x[4] = {x0, x1, x2, x3};
  C o[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    o[r] = tmul(U[4 * r], x[0]);
#pragma unroll
    for (int c = 1; c < 4; ++c) o[r] = tfma(U[4 * r + c], x[c], o[r]);
  }
  x0 = o[0];
  x1 = o[1];
  x2 = o[2];
  x3 = o[3];
}

// Register slots RA < RB, matrix bit 0 <-> RA.
template <int RA, int RB, bool ADJ, class C>
__device__ __forceinline__ void op_u2(C (&v)[16], C (&w)[16], const C* U, uint32_t rm) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    int j = q;
    j = ((j >> RA) << (RA + 1)) | (j & ((1 << RA) - 1));
    j = ((j >> RB) << (RB + 1)) | (j & ((1 << RB) - 1));
    if (!((rm >> j) & 1)) continue;
    const int i1 = j | (1 << RA), i2 = j | (1 << RB), i3 = j | (1 << RA) | (1 << RB);
    u2_quad(v[j], v[i1], v[i2], v[i3], U);
    if (ADJ) u2_quad(w[j], w[i1], w[i2], w[i3], U);
  }
}

template <bool ADJ, class C>
__device__ __forceinline__ void op_phase(C (&v)[16], C (&w)[16], const C* U, uint32_t rm) {
  const C c = U[0];
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    if (!((rm >> j) & 1)) continue;
    v[j] = tmul(c, v[j]);
    if (ADJ) w[j] = tmul(c, w[j]);
  }
}
template <bool ADJ, class C>
__device__ __forceinline__ void op_flip(C (&v)[16], C (&w)[16], uint32_t rm) {
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const bool f = (rm >> j) & 1;
    v[j].x = f ? -v[j].x : v[j].x, v[j].y = f ? -v[j].y : v[j].y;
    if (ADJ) w[j].x = f ? -w[j].x : w[j].x, w[j].y = f ? -w[j].y : w[j].y;
  }
}

// The table index of the op's qubits held by the thread (or outside the
// tile); db: the tile bits of the qubits that may vary over the registers.
template <int ND>
__device__ __forceinline__ uint32_t diag_base(const DevOp* op, uint64_t base, int (&db)[ND]) {
  const int nd = op->nd;
  uint32_t idx = 0;
#pragma unroll
  for (int i = 0; i < ND; ++i) {
    db[i] = i < nd ? op->dbit[i] : -1;
    if (i < nd && db[i] < 0) idx |= (uint32_t)((base >> op->dglob[i]) & 1) << i;
  }
  return idx;
}
// ... and with the bits of tile index t.
template <int ND>
__device__ __forceinline__ uint32_t diag_index(const int (&db)[ND], uint32_t gidx, uint32_t t) {
#pragma unroll
  for (int i = 0; i < ND; ++i)
    if (db[i] >= 0) gidx |= ((t >> db[i]) & 1u) << i;
  return gidx;
}
// The bin idx of a diagonal op's (at most 2) qubits += conj(l) p.
template <class C, class R>
__device__ __forceinline__ void bin_pair(R (&a)[8], uint32_t idx, C l, C p) {
  const R re = fma(l.x, p.x, l.y * p.y), im = fma(l.x, p.y, -l.y * p.x);
#pragma unroll
  for (int b = 0; b < 4; ++b)
    if (idx == (uint32_t)b) {
      a[2 * b] += re;
      a[2 * b + 1] += im;
    }
}
template <class R>
__device__ __forceinline__ void op_accd(const cplx<R> (&v)[16], const cplx<R> (&w)[16], const DevOp* op, uint32_t tthr,
                                        const uint32_t* dep, uint64_t base, R (&a)[8]) {
  int db[2];
  const uint32_t gidx = diag_base(op, base, db);
#pragma unroll
  for (int j = 0; j < 16; ++j) bin_pair(a, diag_index(db, gidx, tthr | dep[j]), w[j], v[j]);
}

// ----------------------------------------------------------------------------- reduced matrices
// A[a][b] += conj(lam_a) psi_b over the op's pairs, after the uncompute.
// KIND & kAccAH: every matrix the partials contract with is anti-Hermitian, so
// only (Im A00, Im A11, Re A01 - Re A10, Im A01 + Im A10) are summed: 12
// instead of 16 products per pair and half the values to reduce.
template <int KIND, class C, class R>
__device__ __forceinline__ void acc_pair(C l0, C l1, C p0, C p1, R (&a)[8]) {
  constexpr int K = KIND & 3;
  if (KIND & kAccAH) {
    if (K != kAccOff) {
      a[0] = fma(l0.x, p0.y, fma(-l0.y, p0.x, a[0]));
      a[1] = fma(l1.x, p1.y, fma(-l1.y, p1.x, a[1]));
    }
    if (K != kAccDiag) {
      a[2] = fma(l0.x, p1.x, fma(l0.y, p1.y, fma(-l1.x, p0.x, fma(-l1.y, p0.y, a[2]))));
      a[3] = fma(l0.x, p1.y, fma(-l0.y, p1.x, fma(l1.x, p0.y, fma(-l1.y, p0.x, a[3]))));
    }
    return;
  }
  if (K != kAccOff) {
    a[0] = fma(l0.x, p0.x, fma(l0.y, p0.y, a[0]));
    a[1] = fma(l0.x, p0.y, fma(-l0.y, p0.x, a[1]));
    a[6] = fma(l1.x, p1.x, fma(l1.y, p1.y, a[6]));
    a[7] = fma(l1.x, p1.y, fma(-l1.y, p1.x, a[7]));
  }
  if (K != kAccDiag) {
    a[2] = fma(l0.x, p1.x, fma(l0.y, p1.y, a[2]));
    a[3] = fma(l0.x, p1.y, fma(-l0.y, p1.x, a[3]));
    a[4] = fma(l1.x, p0.x, fma(l1.y, p0.y, a[4]));
    a[5] = fma(l1.x, p0.y, fma(-l1.y, p0.x, a[5]));
  }
}
template <int RR, bool MASK, int KIND, class R>
__device__ __forceinline__ void op_acc(const cplx<R> (&v)[16], const cplx<R> (&w)[16], uint32_t rm, R (&a)[8]) {
#pragma unroll
  for (int p = 0; p < 8; ++p) {
    const int j0 = pair_lo<RR>(p), j1 = j0 | (1 << RR);
    if (MASK && !((rm >> j0) & 1)) continue;
    acc_pair<KIND>(w[j0], w[j1], v[j0], v[j1], a);
  }
}

// A warp reduce-scatter in FP64 of the first N (4 or 8) values: lane
// i * (32 / N) ends with the total of value i.  Every lane must call it.
template <int N, class R>
__device__ __forceinline__ double warp_scatter(const R (&a)[8]) {
  const int lane = threadIdx.x & 31;
  double x[N];
#pragma unroll
  for (int i = 0; i < N; ++i) x[i] = (double)a[i];
  int o = 16;
#pragma unroll
  for (int k = N; k > 1; k >>= 1, o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < k / 2; ++i) {
      const double keep = up ? x[i + k / 2] : x[i], send = up ? x[i] : x[i + k / 2];
      x[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
#pragma unroll
  for (; o > 0; o >>= 1) x[0] += __shfl_xor_sync(0xffffffffu, x[0], o);
  return x[0];
}
// Thread partials -> the warp's slot row.
template <int N, class R>
__device__ __forceinline__ void flush_acc(const R (&a)[8], double* row) {
  const double u = warp_scatter<N>(a);
  const int lane = threadIdx.x & 31;
  if ((lane & (32 / N - 1)) == 0) row[lane / (32 / N)] += u;
}
// Two ops' first four values at once: nine exchanges instead of twelve and one
// chain of them instead of two; every value's sum has the same order.
template <class R>
__device__ __forceinline__ void flush_two(const R (&a)[4], const R (&b)[8], double* rowa, double* rowb) {
  const R both[8] = {a[0], a[1], a[2], a[3], b[0], b[1], b[2], b[3]};
  const double u = warp_scatter<8>(both);
  const int lane = threadIdx.x & 31, i = lane >> 2;
  if ((lane & 3) == 0) (i < 4 ? rowa : rowb - 4)[i] += u;
}

// ----------------------------------------------------------------------------- a pass
// Per-CTA context of a pass: the tile(s), the accumulation slots and the pass's
// descriptors in shared memory, and the tile counter in the spread (non-tile
// bit) space, base(t + ncta) = ((base | ~mask) + inc) & mask.
template <class R, bool ADJ>
struct TileRun {
  using C = cplx<R>;
  C* psi;
  C* lam;
  C* sp;
  C* sl;
  double* sacc;
  const DevStage* stages;
  const DevOp* ops;
  const C* pool;
  uint64_t base, inc, ntm;
  int64_t namp;  // (the debug build's index limits)
  int T, NW, tlo, thi;
};

// Every thread of the CTA calls it.  stage_pool: the matrices go to shared
// memory with the other descriptors (the interpreter reads them there; a
// compiled pass has them in its parameters).
template <class R, bool ADJ>
__device__ __forceinline__ void tile_begin(TileRun<R, ADJ>& x, const TileItem& it, unsigned char* smem,
                                           uint64_t* s_tile, bool stage_pool) {
  using C = cplx<R>;
  const DevPass& P = it.p;
  const int NT = blockDim.x;
  x.T = 1 << it.M;
  x.NW = NT >> 5;
  x.sp = reinterpret_cast<C*>(smem);
  x.sl = x.sp + (ADJ ? x.T : 0);
  unsigned char* rest = smem + (unsigned long long)(ADJ ? 2 : 1) * x.T * sizeof(C);
  x.sacc = reinterpret_cast<double*>(rest);
  const int nacc = (ADJ ? P.nslots : 0) * x.NW * 8;
  rest += (unsigned long long)nacc * sizeof(double);
  // the pass's descriptors (stages, ops, matrices), 16-byte words
  const int n1 = (int)(sizeof(DevStage) / 16) * (P.stage_end - P.stage_begin),
            n2 = n1 + (int)(sizeof(DevOp) / 16) * P.nops,
            n3 = n2 + (stage_pool ? (int)((sizeof(C) * P.npool + 15) / 16) : 0);
  const int4* s1 = reinterpret_cast<const int4*>((const DevStage*)it.stages + P.stage_begin);
  const int4* s2 = reinterpret_cast<const int4*>(it.ops) - n1;
  const int4* s3 = reinterpret_cast<const int4*>(it.pool) - n2;
  int4* d = reinterpret_cast<int4*>(rest);
#pragma unroll 4
  for (int i = threadIdx.x; i < n3; i += NT) d[i] = __ldg(i < n1 ? s1 + i : (i < n2 ? s2 + i : s3 + i));
  for (int i = threadIdx.x; i < nacc; i += NT) x.sacc[i] = 0;
  if (threadIdx.x == NT - 1) {
    // the first tile's base (tile index spread over the non-tile qubits) and
    // the increment for ncta tiles in the same spread form
    uint64_t mm = P.nontile_mask, b0 = 0, inc = 0;
    uint32_t t = blockIdx.x, s = (uint32_t)it.ncta;
    while (mm) {
      const uint64_t low = mm & (~mm + 1);
      if (t & 1) b0 |= low;
      if (s & 1) inc |= low;
      t >>= 1;
      s >>= 1;
      mm ^= low;
    }
    s_tile[0] = b0;
    s_tile[1] = inc;
  }
  __syncthreads();
  x.stages = reinterpret_cast<const DevStage*>(rest);
  x.ops = reinterpret_cast<const DevOp*>(rest + 16ull * n1);
  x.pool = reinterpret_cast<const C*>(rest + 16ull * n2);
  x.base = s_tile[0];
  x.inc = s_tile[1];
  x.ntm = P.nontile_mask;
  x.namp = P.ntiles << it.M;
  x.psi = (C*)it.psi;
  x.lam = (C*)it.lam;
  x.tlo = threadIdx.x & 15;
  x.thi = threadIdx.x >> 4;
}
template <class R, bool ADJ>
__device__ __forceinline__ void tile_advance(TileRun<R, ADJ>& x) {
  x.base = ((x.base | ~x.ntm) + x.inc) & x.ntm;
}

// A stage's amplitudes: from HBM (the pass's first stage) or shared memory,
// and back (HBM after its last).  swm / gdep: the stage's tables, in shared
// memory or as constants.
template <class R, bool ADJ, class S32, class S64>
__device__ __forceinline__ void tile_load(const TileRun<R, ADJ>& x, const DevStage* S, bool first, cplx<R> (&v)[16],
                                          cplx<R> (&w)[16], const S32& swm, const S64& gdep) {
  if (first) {
    const int64_t g0 = (int64_t)x.base + S->gthr[0][x.tlo] + S->gthr[1][x.thi];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int64_t gi = g0 + gdep[j];
      if (!VQC_DCHECK(gi, x.namp)) continue;
      v[j] = x.psi[gi];
      if (ADJ) w[j] = x.lam[gi];
    }
  } else {
    const uint32_t sw = S->swt[0][x.tlo] ^ S->swt[1][x.thi];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const uint32_t t = sw ^ swm[j];
      if (!VQC_DCHECK(t, x.T)) continue;
      v[j] = x.sp[t];
      if (ADJ) w[j] = x.sl[t];
    }
  }
}
// Ends the stage: a thread stores exactly the amplitudes it loaded, so the only
// hazard is the next stage (or tile) reading what another thread stored; cta =
// false: it keeps the warp index on the same tile bits, a warp barrier does.
template <class R, bool ADJ, class S32, class S64>
__device__ __forceinline__ void tile_store(const TileRun<R, ADJ>& x, const DevStage* S, bool last,
                                           const cplx<R> (&v)[16], const cplx<R> (&w)[16], const S32& swm,
                                           const S64& gdep, bool cta) {
  if (last) {
    const int64_t g0 = (int64_t)x.base + S->gthr[0][x.tlo] + S->gthr[1][x.thi];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int64_t gi = g0 + gdep[j];
      if (!VQC_DCHECK(gi, x.namp)) continue;
      x.psi[gi] = v[j];
      if (ADJ) x.lam[gi] = w[j];
    }
  } else {
    const uint32_t sw = S->swt[0][x.tlo] ^ S->swt[1][x.thi];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const uint32_t t = sw ^ swm[j];
      if (!VQC_DCHECK(t, x.T)) continue;
      x.sp[t] = v[j];
      if (ADJ) x.sl[t] = w[j];
    }
  }
  if (cta)
    __syncthreads();
  else
    __syncwarp();
}

template <class R, bool ADJ>
__device__ __forceinline__ double* tile_slot(const TileRun<R, ADJ>& x, int slot) {
  return x.sacc + ((unsigned long long)slot * x.NW + (threadIdx.x >> 5)) * 8;
}
// Per-warp slot rows -> this CTA's partials row (fixed order).
template <class R, bool ADJ>
__device__ __forceinline__ void tile_end(const TileRun<R, ADJ>& x, const TileItem& it) {
  const int nslots = ADJ ? it.p.nslots : 0;
  if (nslots == 0) return;
  __syncthreads();
  for (int i = threadIdx.x; i < nslots * 8; i += blockDim.x) {
    const int slot = i >> 3, val = i & 7;
    double s = 0;
    for (int wp = 0; wp < x.NW; ++wp) s += x.sacc[((unsigned long long)slot * x.NW + wp) * 8 + val];
    it.partials[((unsigned long long)blockIdx.x * nslots + slot) * 8 + val] = s;
  }
}

}  // namespace vqc
