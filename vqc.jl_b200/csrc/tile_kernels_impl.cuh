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
// shared memory a 12-qubit FP64 reverse pass takes 66 us (93), a 17-qubit FP32
// one 46 us (59), the serving loop's reverse launches 68 us (97), a 17-qubit FP32
// forward pass 28 us (31).  Bound by latency: a tile's few warps, each op's
// decoding, loads and chain of FMAs one after another.
#pragma once

#include "engine.h"
#include "subspace.cuh"
#include "tile_plan.cuh"
#include "tile_f32.cuh"
#include "tile_ops.cuh"

namespace vqc {

// ----------------------------------------------------------------------------- ops in shared memory
constexpr int kAccNone = 3;  // (between the kinds of kAcc*: 0-2, 4-6)

// The second 16-byte word of an op (DevOp: first, step, target, slot).
struct OpWord {
  uint32_t first, step[3], target[2];
  int slot;
  __device__ __forceinline__ explicit OpWord(int4 w) {
    first = (uint32_t)w.x & 0xffffu, step[0] = (uint32_t)w.x >> 16;
    step[1] = (uint32_t)w.y & 0xffffu, step[2] = (uint32_t)w.y >> 16;
    target[0] = (uint32_t)w.z & 0xffffu, target[1] = (uint32_t)w.z >> 16;
    slot = w.w;
  }
};
template <class C>
__device__ __forceinline__ C& at(unsigned char* tile, uint32_t byte) {
  return *reinterpret_cast<C*>(tile + byte);
}

// N pairs, at a ^ off[i] and the same ^ t (bytes): all loads first (a pair's
// chain of dependent FMAs is longer than a load, and a store bars the next load
// from moving up), U on psi and lambda, the pairs' terms of the reduced matrix
// in order, all stores.
template <int N, int FORM, int ACC, bool ADJ, class R>
__device__ __forceinline__ void pair_group(unsigned char* sp, unsigned char* sl, uint32_t a, uint32_t t,
                                           const uint32_t (&off)[4], const cplx<R> (&u)[4], R (&acc)[8]) {
  using C = cplx<R>;
  C p0[N], p1[N], l0[N], l1[N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const uint32_t b = a ^ off[i], c = b ^ t;
    p0[i] = at<C>(sp, b), p1[i] = at<C>(sp, c);
    if (ADJ) l0[i] = at<C>(sl, b), l1[i] = at<C>(sl, c);
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
    const uint32_t b = a ^ off[i], c = b ^ t;
    at<C>(sp, b) = p0[i], at<C>(sp, c) = p1[i];
    if (ADJ) at<C>(sl, b) = l0[i], at<C>(sl, c) = l1[i];
  }
}

// The op's pairs in ascending order of their free bits (the compiled passes
// sum in the same order), four at a time where there are four.
template <int FORM, int ACC, bool ADJ, class R>
__device__ __forceinline__ void pair_loop(unsigned char* sp, unsigned char* sl, uint32_t a, const OpWord& op,
                                          int nfree, const cplx<R>* U, R (&acc)[8]) {
  const cplx<R> u[4] = {U[0], U[1], U[2], U[3]};
  const uint32_t t = op.target[0], off[4] = {0u, op.step[0], op.step[1], op.step[0] ^ op.step[1]};
  if (nfree >= 2) {
    pair_group<4, FORM, ACC, ADJ, R>(sp, sl, a, t, off, u, acc);
    if (nfree == 3) pair_group<4, FORM, ACC, ADJ, R>(sp, sl, a ^ op.step[2], t, off, u, acc);
  } else {
    pair_group<1, FORM, ACC, ADJ, R>(sp, sl, a, t, off, u, acc);
    if (nfree == 1) pair_group<1, FORM, ACC, ADJ, R>(sp, sl, a ^ off[1], t, off, u, acc);
  }
}

// One switch over the matrix form and what the op sums of the reduced matrix.
template <bool ADJ, class R>
__device__ __forceinline__ void pair_switch(int form, int acck, unsigned char* sp, unsigned char* sl, uint32_t a,
                                            const OpWord& op, int nfree, const cplx<R>* U, R (&acc)[8]) {
#define VQC_FORMS(X, K)                                                                                        \
  X(kFormGen, K) X(kFormRI, K) X(kFormReal, K) X(kFormDiag, K) X(kFormSwap, K) X(kFormUD, K) X(kFormRC, K) \
  X(kFormOff, K) X(kFormId, K)
#define VQC_CASE(F, K)                                                                          \
  case F + kForms * K:                                                                          \
    if constexpr (interpreted_form<R>(F) == F) pair_loop<F, K, ADJ, R>(sp, sl, a, op, nfree, U, acc); \
    break;
  if constexpr (ADJ) {
    switch (form + kForms * acck) {
      VQC_FORMS(VQC_CASE, kAccFull)
      VQC_FORMS(VQC_CASE, kAccOff)
      VQC_FORMS(VQC_CASE, kAccDiag)
      VQC_FORMS(VQC_CASE, (kAccAH | kAccFull))
      VQC_FORMS(VQC_CASE, (kAccAH | kAccOff))
      VQC_FORMS(VQC_CASE, (kAccAH | kAccDiag))
      VQC_FORMS(VQC_CASE, kAccNone)
      default: break;
    }
  } else {
    switch (form + kForms * kAccNone) {
      VQC_FORMS(VQC_CASE, kAccNone)
      default: break;
    }
  }
#undef VQC_CASE
#undef VQC_FORMS
}

template <class R>
__device__ __forceinline__ void quad_loop(unsigned char* s, uint32_t a, const OpWord& op, int nfree,
                                          const cplx<R>* U) {
  using C = cplx<R>;
  const uint32_t ta = op.target[0], tb = op.target[1];
  for (int k = 0; k < (1 << nfree); ++k) {
    const uint32_t b = a ^ ((k & 1) ? op.step[0] : 0u) ^ ((k & 2) ? op.step[1] : 0u);
    C x0 = at<C>(s, b), x1 = at<C>(s, b ^ ta), x2 = at<C>(s, b ^ tb), x3 = at<C>(s, b ^ ta ^ tb);
    u2_quad(x0, x1, x2, x3, U);
    at<C>(s, b) = x0, at<C>(s, b ^ ta) = x1, at<C>(s, b ^ tb) = x2, at<C>(s, b ^ ta ^ tb) = x3;
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
  unsigned char* bp = reinterpret_cast<unsigned char*>(sp);
  unsigned char* bl = reinterpret_cast<unsigned char*>(sl);
  for (int64_t tile = blockIdx.x; tile < it.p.ntiles; tile += it.ncta) {
    for (int s = 0; s < nstages; ++s) {
      const DevStage* S = x.stages + s;
      const uint32_t tthr = S->thr[0][x.tlo] | S->thr[1][x.thi], sw = S->swt[0][x.tlo] ^ S->swt[1][x.thi];
      const uint32_t swb = sw * (uint32_t)sizeof(C);
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
      int o = S->op_begin, held = -1;  // held: the slot of an op whose sums wait for a second op's
      R ha[4];
      const int4* words = reinterpret_cast<const int4*>(x.ops + o);
      // read one op ahead, never past the pass's ops: a coalesced end stage has none,
      // and behind them the launch may have asked for one matrix's word only
      int4 w0 = make_int4(0, 0, 0, 0), w1 = w0;
      if (o < oe && VQC_DCHECK(o, it.p.nops)) w0 = words[0], w1 = words[1];
#pragma unroll 1
      for (; o < oe; ++o) {
        const DevOp* op = x.ops + o;
        const int4 cur = w0;
        const OpWord ow(w1);
        words += sizeof(DevOp) / 16;
        if (o + 1 < oe && VQC_DCHECK(o + 1, it.p.nops)) w0 = words[0], w1 = words[1];
        const int code = cur.x, sel = (code >> kSelShift) & 127;
        if (code & kCodeGCtl) {  // a control on a non-tile qubit: uniform over the tile
          if ((x.base & op->gmask) != op->gval) continue;
        }
        // controls on thread bits: one test per op (it may differ between the
        // lanes of a warp: the warp-wide reduction below runs outside it)
        const bool run = !(code & kCodeCtl) || (tthr & (uint32_t)cur.z) == (uint32_t)cur.w;
        const bool acc = ADJ && (code & kCodeAcc);
        const C* U = x.pool + cur.y;
        const int kind = acc_kind_of(code), nf = op_free(code);
        R a[8];
        if (ADJ) {
#pragma unroll
          for (int i = 0; i < 8; ++i) a[i] = R(0);
        }
        if (run) {
          const uint32_t t = swb ^ ow.first;
          if (sel < kSelU2) {
            if (VQC_DCHECK(t ^ ow.target[0], sizeof(C) * x.T))
              pair_switch<ADJ, R>(sel >> 3, acc ? kind : kAccNone, bp, bl, t, ow, nf, U, a);
          } else if (sel < kSelPhase) {
            quad_loop<R>(bp, t, ow, nf, U);
            if (ADJ) quad_loop<R>(bl, t, ow, nf, U);
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
          if (!(kind & kAccAH)) {
            flush_acc<8>(a, tile_slot(x, ow.slot));
          } else if (held < 0) {
            held = ow.slot;
#pragma unroll
            for (int i = 0; i < 4; ++i) ha[i] = a[i];
          } else {
            flush_two(ha, a, tile_slot(x, held), tile_slot(x, ow.slot));
            held = -1;
          }
        }
      }
      if (ADJ && held >= 0) {
        R a[8] = {ha[0], ha[1], ha[2], ha[3], R(0), R(0), R(0), R(0)};
        flush_acc<4>(a, tile_slot(x, held));
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

// Resident CTAs the registers are budgeted for: forward what the tiles in shared
// memory admit (32 KiB each plus descriptors); reverse two, without spills (at
// three a 17-qubit FP32 reverse pass takes 70 against 46 us).
template <class R, bool ADJ>
struct TileBounds {
  static constexpr int nt = sizeof(R) == 4 ? 256 : 128, nb = ADJ ? 2 : 5;
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
