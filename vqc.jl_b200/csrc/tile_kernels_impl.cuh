// Device code of the fused tile engine: the classic tile body (FP64 passes,
// and FP32 passes that are not compiled at run time) and its kernels k_tile /
// k_tile_batch.  The kernels are instantiated in the tile_inst_*.cu
// translation units (compiled in parallel); the planner in fused.cu sees only
// their declarations (tile_kernels.cuh).
//
// The body interprets a pass with the tile in shared memory.  A stage gives
// every thread 16 amplitudes of its own (4 tile bits), so its ops need no
// barrier; each op loops over the thread's amplitude pairs, two loads, the
// 2x2, two stores, at addresses that are XORs of per-op offsets.  What the op
// does (matrix form, which products of the reduced matrix it sums) is one
// switch per op; which bits it acts on is data.
//
// Holding the 16 amplitudes in registers instead needs a variant per target
// bit, and every switch then moves all of them between the variants' register
// assignments: 1,360 instructions per op of a reverse FP64 pass, 395 of them
// arithmetic (counted on 2^22 amplitudes), with the FP64 pipe at 25 %.  In
// shared memory a 12-qubit FP64 reverse pass takes 73 us (93), a 17-qubit FP32
// one 50 us (59), the serving loop's reverse launches 66 us (97); forward passes
// are even (41, 31 and 57 us).
#pragma once

#include "engine.h"
#include "subspace.cuh"
#include "tile_plan.cuh"
#include "tile_f32.cuh"
#include "tile_ops.cuh"

namespace vqc {

// ----------------------------------------------------------------------------- ops in shared memory
constexpr int kAccNone = 8;  // (after the kinds of kAcc*)

// N pairs, at a ^ off[i] and the same ^ t: all loads first (a pair's chain of
// dependent FMAs is longer than a load, and a store bars the next load from
// moving up), U on psi and lambda, the pairs' terms of the reduced matrix in
// order, all stores.
template <int N, int FORM, int ACC, bool ADJ, class R>
__device__ __forceinline__ void pair_group(cplx<R>* sp, cplx<R>* sl, uint32_t a, uint32_t t, const uint32_t (&off)[4],
                                           const cplx<R> (&u)[4], R (&acc)[8]) {
  using C = cplx<R>;
  C p0[N], p1[N], l0[N], l1[N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const uint32_t b = a ^ off[i];
    p0[i] = sp[b], p1[i] = sp[b ^ t];
    if (ADJ) l0[i] = sl[b], l1[i] = sl[b ^ t];
  }
#pragma unroll
  for (int i = 0; i < N; ++i) {
    u1_apply<FORM>(p0[i], p1[i], u);
    if (ADJ) {
      u1_apply<FORM>(l0[i], l1[i], u);
      if (ACC != kAccNone) acc_pair<ACC>(l0[i], l1[i], p0[i], p1[i], acc);
    }
  }
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const uint32_t b = a ^ off[i];
    sp[b] = p0[i], sp[b ^ t] = p1[i];
    if (ADJ) sl[b] = l0[i], sl[b ^ t] = l1[i];
  }
}

// The op's pairs in ascending order of their free bits (the compiled passes
// sum in the same order), four at a time where there are four.
template <int FORM, int ACC, bool ADJ, class R>
__device__ __forceinline__ void pair_loop(cplx<R>* sp, cplx<R>* sl, uint32_t a, const DevOp* op, int nfree,
                                          const cplx<R>* U, R (&acc)[8], [[maybe_unused]] int T) {
  const cplx<R> u[4] = {U[0], U[1], U[2], U[3]};
  const uint32_t t = op->target[0], f0 = op->step[0], f1 = op->step[1];
  const uint32_t off[4] = {0u, f0, f1, f0 ^ f1};
  if (!VQC_DCHECK(a ^ t, T)) return;
  if (nfree >= 2) {
    pair_group<4, FORM, ACC, ADJ, R>(sp, sl, a, t, off, u, acc);
    if (nfree == 3) pair_group<4, FORM, ACC, ADJ, R>(sp, sl, a ^ op->step[2], t, off, u, acc);
  } else {
    pair_group<1, FORM, ACC, ADJ, R>(sp, sl, a, t, off, u, acc);
    if (nfree == 1) pair_group<1, FORM, ACC, ADJ, R>(sp, sl, a ^ f0, t, off, u, acc);
  }
}
template <int FORM, bool ADJ, class R>
__device__ __forceinline__ void pair_acc(int acck, cplx<R>* sp, cplx<R>* sl, uint32_t a, const DevOp* op, int nfree,
                                         const cplx<R>* U, R (&acc)[8], int T) {
  if constexpr (ADJ) {
    switch (acck) {
      case kAccFull: pair_loop<FORM, kAccFull, ADJ, R>(sp, sl, a, op, nfree, U, acc, T); return;
      case kAccOff: pair_loop<FORM, kAccOff, ADJ, R>(sp, sl, a, op, nfree, U, acc, T); return;
      case kAccDiag: pair_loop<FORM, kAccDiag, ADJ, R>(sp, sl, a, op, nfree, U, acc, T); return;
      case kAccAH | kAccFull: pair_loop<FORM, kAccAH | kAccFull, ADJ, R>(sp, sl, a, op, nfree, U, acc, T); return;
      case kAccAH | kAccOff: pair_loop<FORM, kAccAH | kAccOff, ADJ, R>(sp, sl, a, op, nfree, U, acc, T); return;
      case kAccAH | kAccDiag: pair_loop<FORM, kAccAH | kAccDiag, ADJ, R>(sp, sl, a, op, nfree, U, acc, T); return;
      default: break;
    }
  }
  pair_loop<FORM, kAccNone, ADJ, R>(sp, sl, a, op, nfree, U, acc, T);
}

template <class R>
__device__ __forceinline__ void quad_loop(cplx<R>* s, uint32_t a, const DevOp* op, int nfree, const cplx<R>* U) {
  using C = cplx<R>;
  const uint32_t ta = op->target[0], tb = op->target[1];
  for (int k = 0; k < (1 << nfree); ++k) {
    const uint32_t b = a ^ ((k & 1) ? op->step[0] : 0u) ^ ((k & 2) ? op->step[1] : 0u);
    C x0 = s[b], x1 = s[b ^ ta], x2 = s[b ^ tb], x3 = s[b ^ ta ^ tb];
    u2_quad(x0, x1, x2, x3, U);
    s[b] = x0, s[b ^ ta] = x1, s[b ^ tb] = x2, s[b ^ ta ^ tb] = x3;
  }
}

// A phase (or a flip of sign) on the amplitudes in rmask.
template <bool FLIP, class R>
__device__ __forceinline__ void phase_loop(cplx<R>* s, uint32_t sw, const DevStage* S, uint32_t rm, const cplx<R>* U) {
  using C = cplx<R>;
  for (uint32_t m = rm; m; m &= m - 1) {
    const uint32_t t = sw ^ S->swm[__ffs(m) - 1];
    const C x = s[t];
    if (FLIP)
      s[t] = mkc<R>(-x.x, -x.y);
    else
      s[t] = tmul(U[0], x);
  }
}
template <bool ADJ, class R>
__device__ __forceinline__ void diag_loop(cplx<R>* sp, cplx<R>* sl, uint32_t sw, const DevStage* S, const DevOp* op,
                                          const cplx<R>* U, uint32_t tthr, uint64_t base) {
  int db[5];
  const uint32_t gidx = diag_base(op, base, db);
  for (int j = 0; j < 16; ++j) {
    const uint32_t i = diag_index(db, gidx, tthr | S->dep[j]), t = sw ^ S->swm[j];
    sp[t] = tmul(U[i], sp[t]);
    if (ADJ) sl[t] = tmul(U[i], sl[t]);
  }
}
template <class R>
__device__ __forceinline__ void accd_loop(const cplx<R>* sp, const cplx<R>* sl, uint32_t sw, const DevStage* S,
                                          const DevOp* op, uint32_t tthr, uint64_t base, R (&a)[8]) {
  int db[2];
  const uint32_t gidx = diag_base(op, base, db);
  for (int j = 0; j < 16; ++j) {
    const uint32_t i = diag_index(db, gidx, tthr | S->dep[j]), t = sw ^ S->swm[j];
    bin_pair(a, i, sl[t], sp[t]);
  }
}

// ----------------------------------------------------------------------------- the tile loop
template <class R, bool ADJ>
__device__ __forceinline__ void tile_body(const TileItem& it) {
  using C = cplx<R>;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ uint64_t s_tile[2];
  TileRun<R, ADJ> x;
  tile_begin<R, ADJ>(x, it, smem, s_tile, true);
  const int nstages = it.p.stage_end - it.p.stage_begin;
  C* sp = x.sp;
  C* sl = x.sl;
  for (int64_t tile = blockIdx.x; tile < it.p.ntiles; tile += it.ncta) {
    for (int s = 0; s < nstages; ++s) {
      const DevStage* S = x.stages + s;
      const uint32_t tthr = S->thr[0][x.tlo] | S->thr[1][x.thi], sw = S->swt[0][x.tlo] ^ S->swt[1][x.thi];
      if (s == 0) {
        C v[16], w[16];
        tile_load<R, ADJ>(x, S, true, v, w, S->swm, S->gdep);
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const uint32_t t = sw ^ S->swm[j];
          if (!VQC_DCHECK(t, x.T)) continue;
          sp[t] = v[j];
          if (ADJ) sl[t] = w[j];
        }
      }
      const int oe = S->op_end;
      int o = S->op_begin;
      int4 hd = o < oe ? *reinterpret_cast<const int4*>(x.ops + o) : make_int4(0, 0, 0, 0);
#pragma unroll 1
      for (; o < oe; ++o) {
        const DevOp* op = x.ops + o;
        const int4 cur = hd;
        if (o + 1 < oe) hd = *reinterpret_cast<const int4*>(op + 1);
        const int code = cur.x, sel = (code >> kSelShift) & 127;
        if (code & kCodeGCtl) {  // a control on a non-tile qubit: uniform over the tile
          if ((x.base & op->gmask) != op->gval) continue;
        }
        // controls on thread bits: one test per op (it may differ between the
        // lanes of a warp: the warp-wide reduction below runs outside it)
        const bool run = !(code & kCodeCtl) || (tthr & (uint32_t)cur.z) == (uint32_t)cur.w;
        const bool acc = ADJ && (code & kCodeAcc);
        const C* U = x.pool + cur.y;
        const int kind = acc_kind_of(code), acck = acc ? kind : kAccNone, nf = op_free(code);
        R a[8];
        if (ADJ) {
#pragma unroll
          for (int i = 0; i < 8; ++i) a[i] = R(0);
        }
        if (run) {
          const uint32_t t = sw ^ op->first;
          if (sel < kSelU2) {
            switch (sel >> 3) {
              case kFormRI: pair_acc<kFormRI, ADJ, R>(acck, sp, sl, t, op, nf, U, a, x.T); break;
              case kFormReal: pair_acc<kFormReal, ADJ, R>(acck, sp, sl, t, op, nf, U, a, x.T); break;
              case kFormDiag: pair_acc<kFormDiag, ADJ, R>(acck, sp, sl, t, op, nf, U, a, x.T); break;
              case kFormSwap: pair_acc<kFormSwap, ADJ, R>(acck, sp, sl, t, op, nf, U, a, x.T); break;
              case kFormUD: pair_acc<kFormUD, ADJ, R>(acck, sp, sl, t, op, nf, U, a, x.T); break;
              case kFormRC: pair_acc<kFormRC, ADJ, R>(acck, sp, sl, t, op, nf, U, a, x.T); break;
              case kFormOff: pair_acc<kFormOff, ADJ, R>(acck, sp, sl, t, op, nf, U, a, x.T); break;
              case kFormId:
                if (acc) pair_acc<kFormId, ADJ, R>(acck, sp, sl, t, op, nf, U, a, x.T);
                break;
              default: pair_acc<kFormGen, ADJ, R>(acck, sp, sl, t, op, nf, U, a, x.T); break;
            }
          } else if (sel < kSelPhase) {
            quad_loop<R>(sp, t, op, nf, U);
            if (ADJ) quad_loop<R>(sl, t, op, nf, U);
          } else if (sel == kSelFlip) {
            phase_loop<true, R>(sp, sw, S, (uint32_t)op->rmask, U);
            if (ADJ) phase_loop<true, R>(sl, sw, S, (uint32_t)op->rmask, U);
          } else if (sel == kSelPhase) {
            phase_loop<false, R>(sp, sw, S, (uint32_t)op->rmask, U);
            if (ADJ) phase_loop<false, R>(sl, sw, S, (uint32_t)op->rmask, U);
          } else if (sel == kSelDiag) {
            diag_loop<ADJ, R>(sp, sl, sw, S, op, U, tthr, x.base);
          } else if (ADJ) {
            accd_loop<R>(sp, sl, sw, S, op, tthr, x.base, a);
          }
        }
        if (acc) {
          if (kind & kAccAH)
            flush_acc<4>(a, tile_slot(x, op->slot));
          else
            flush_acc<8>(a, tile_slot(x, op->slot));
        }
      }
      if (s == nstages - 1) {
        C v[16], w[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const uint32_t t = sw ^ S->swm[j];
          if (!VQC_DCHECK(t, x.T)) continue;
          v[j] = sp[t];
          if (ADJ) w[j] = sl[t];
        }
        tile_store<R, ADJ>(x, S, true, v, w, S->swm, S->gdep, S->cta);
      } else if (S->cta) {
        __syncthreads();
      } else {
        __syncwarp();
      }
    }
    tile_advance(x);
  }
  tile_end(x, it);
}

// Resident CTAs: what the tiles in shared memory admit (32 KiB, reverse 64 KiB,
// plus descriptors), registers budgeted for it.
template <class R, bool ADJ>
struct TileBounds {
  static constexpr int nt = sizeof(R) == 4 ? 256 : 128, nb = ADJ ? 3 : 5;
};

template <class R, bool ADJ>
__global__ void __launch_bounds__(TileBounds<R, ADJ>::nt, TileBounds<R, ADJ>::nb)
    k_tile(const __grid_constant__ TileItem item) {
  tile_body<R, ADJ>(item);
}

template <class R, bool ADJ>
__global__ void __launch_bounds__(TileBounds<R, ADJ>::nt, TileBounds<R, ADJ>::nb)
    k_tile_batch(const TileItem* __restrict__ items) {
  const TileItem it = items[blockIdx.y];
  if ((int)blockIdx.x >= it.ncta) return;
  tile_body<R, ADJ>(it);
}

// The FP32 packed body (tile_f32.cuh) on a plan laid out for it (lane bit in
// every stage, DevStageF): the interpreted form of the run-time compiled
// passes, for a pass whose compiled kernel is missing.
template <int M, bool ADJ>
__global__ void __launch_bounds__(1 << (M - kRegBits), ADJ ? 2 : 3)
    k_tile_packed(const __grid_constant__ TileItem it) {
  f32t::tile_body<M, ADJ, true>((float2*)it.psi, (float2*)it.lam, it.pass, (const DevStageF*)it.stages, it.ops,
                                (const float2*)it.pool, it.partials, it.ncta);
}

}  // namespace vqc
