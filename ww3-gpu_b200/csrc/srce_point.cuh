// ww3-gpu_b200/csrc/srce_point.cuh
// W3SRCE (the dynamic-substep source-term integration of a sea point: ST4 + the DIA + W3SLN1,
// W3SBT1, W3SDB1, MLIM, SEED) for a CTA that integrates several points side by side, written
// once for the device and the host.
//
// Reference: ww3-gpu kokkos/src/ww_kokkos/srce_kernel.hpp:140-583 (SrcePoint: init, step_a,
// dia, step_c, finish; WW3 w3srcemd.F90:869-2350 at 03adda91), st4_sin4.hpp:69-630,
// st4_sds4.hpp:120-745, st4_spr4.hpp:40-160, srce_db1.hpp:33-150, srce_bt1.hpp (W3SBT1),
// srce_ln1.hpp (W3SLN1), snl1_team.hpp:351-497 (the DIA in its row-shift form). Each statement
// keeps the reference's operand order; MAX/MIN sites keep its operand order (mx(a,b) = a > b ? a
// : b, mn(a,b) = a < b ? a : b); every ordered sum is one running sum in the reference's order.
//
// Why several points per CTA. A substep is a few hundred thousand instructions that any thread
// can do and some fifteen ordered chains (sums over 1296 bins, Newton steps, the stress scan
// over frequency, the 50-step tail) that one thread does. With one point per CTA the chains leave
// 127 of 128 threads at a barrier and the four CTAs of an SM evict each other's code from the
// instruction cache: on B200, 36 x 36 bins, 9,520 points took 422 ms and a launch of 5 points 24.8 ms;
// in slots 102 ms and 4.5 ms. What bounds it now: instruction issue (about 2 of 4 per cycle) and fetch (two
// CTAs of four slots per SM, in two phases at a time, ran 7 % longer than one of eight, three of three
// slots 60 % longer; both measured with fewer registers per thread than now).
// Here a CTA holds up to kSlots points in slots. A phase is either a loop over all (slot, bin) or
// (slot, frequency) pairs by all warps, or a set of roles: role r is warp r, its lane k the chain of
// slot k, so the chains of all slots and roles run at the same time and one instruction serves
// every slot. All warps of the CTA are in the same phase, so the code they fetch is the same.
//
// A slot's point moves through states, so that a slot is refilled as soon as its point is done:
// kFresh1 (first W3SPR4 and W3SIN4 of W3SRCE's initialisation), kFresh2 (its second W3SPR4 and the
// first step's W3SIN4), kRun (whole steps). Points in different states share the calls of W3SPR4
// and W3SIN4 of one trip of the loop.
//
// Working set (floats): per slot in shared memory SPEC, LLWS (bytes), WN1 CG1 DAM and three NK
// arrays fixed for the point, CBETA, W3SLN1's two arrays; one transient region shared by the
// phases (the DIA's UE, SA1, SA2 of a few slots at a time; W3SDS4's BTH / BRLAMBDA and NK arrays;
// the terms of the closing sums; W3SIN4's stress terms). Per slot in global scratch, read and written
// by parallel loops only: SPECINIT VDIN VSNL VDNL VSDS VDDS VSDB and the DIA's DA arrays.
#pragma once

#include "snl1_kernel.cuh"
#include "st4_point.cuh"

namespace wwb {
namespace pt {

WWB_PD float mx(float a, float b) { return a > b ? a : b; }
WWB_PD float mn(float a, float b) { return a < b ? a : b; }

/// W3SRCE's own grid arrays (ww_srce_init), 0-based: sig[ik] = SIG(IK+1) etc.
struct SrceGrid {
  const float *sig, *dden, *ecos, *esin;
  const int* mapwn;
};

/// Per-point inputs and the step's flags.
struct SrceIn {
  int it, inflags24, flogrd57, flogrd58;
  float d_inp, u10abs, u10dir, as, ice, dtg, dair, coef;
};

/// Points a CTA integrates side by side: a chain phase costs the same for eight as for one, and their
/// working sets (22 KB each at 36 x 36) fill the SM's shared memory. One CTA of four per SM ran 167 ms for
/// 9,520 points where two of four ran 133; one of eight ran 98.7 where two of four ran 106 (taken on the
/// way here, with 768 threads; now 102).
constexpr int kSlots = 8;

enum SlotState : int { kIdle = 0, kFresh1 = 1, kFresh2 = 2, kRun = 3, kDone = 4 };

/// A point's scalars, shared by the CTA. r holds W3SPR4's outputs under W3SRCE's names
/// (r.ustar = USTAR, r.usdir = USTDIR, r.wnmean = WNMEAN, ...).
struct SrceSh {
  Spr4Out r;
  float tauwx, tauwy, dtdyn, fcut, tauox, tauoy, tauwix, tauwiy, tauwnx, tauwny, phiaw, tws,
      phioc, phibbl, phice, tauocx, tauocy, fpi;
  int shave;
  float whitecap[4], taubbl[2], tauice[2];
  SrceIn in;
  float depth, drat, icescaleln, icescalein, icescalenl, icescaleds;
  float fage, fhigh, dttot, dt, tauwax, tauway, vddb, afilt, mlim, cons;
  int nsteps, nkh, nkh1, nspech, nscut, state, early, done;
  unsigned vmin;      ///< bits of the running MIN of the time-step limits (values >= 0)
  float chains[3];    ///< W3SPR4's ELCS, ELSN, AMAX
  float c0;           ///< the tail level's factor (:880), a function of the point's CG
  float stress[2], usdirpl, levtail0, tauhf;  ///< W3SIN4's closing part
  // W3SIN4
  float fwuorb, pturb, pvisc, fu, fud, ustarsigma, const1;  ///< fwuorb = FW * UORB
  float ust, taux, tauy, cosu, sinu, ustp, cosw, sinw;  ///< cosw, sinw: of the wind direction
  float sums[4];      ///< running STRESS (x, y) and STRESSN (x, y) of one pass
  float ss[3][2], sn[3][2];
  int scan_par;       ///< the stress scan's frequencies are independent of one another
  // W3SDS4, W3SLN1
  float facturb, cosus, sinus;
};

/// Offsets (in floats) of the working set; see the file header.
struct SrceLayout {
  int nspec, nk, nth;
  unsigned nth_magic;  ///< i / nth = umulhi(i, nth_magic) for the bins' range
  // shared: what all slots read, then per slot (stride ws), then the transient region
  int pwsig, pwdir, tail, ec, es, common;
  int ws, spec, llws, wn1, cg1, dam, pwwn, mft, cbeta, wnf, dirf, jt;  ///< jt: the tail's arrays over its steps
  int tslot;           ///< transient floats a slot needs outside the DIA
  int dia;             ///< transient floats of one slot's DIA
  // global scratch per slot
  int specinit, vdin, vsnl, vdnl, vsds, vdds, vsdb, da, alen;
  int total_s;         ///< floats of shared memory with one slot
  int total_g;         ///< floats of global scratch per slot
};

/// Floats of an array over the tail's steps.
constexpr int kJtot4 = (kJtot + 3) & ~3;
/// NK arrays a phase of W3SDS4 / W3SPR4 / W3SIN4 keeps in the transient region.
constexpr int kNkWork = 20;

/// Floats of shared memory of a CTA with ns slots.
WWB_PD int srce_trans_floats(const SrceLayout& L, int ns) {
  return ns * L.tslot > L.dia ? ns * L.tslot : L.dia;
}
WWB_PD int srce_shared_floats(const SrceLayout& L, int ns) {
  return L.common + ns * L.ws + srce_trans_floats(L, ns);
}

inline SrceLayout srce_layout(const st4::Params& q, const Snl1Dev& n) {
  SrceLayout L{};
  const int ns = q.nspec, nk = q.nk, nth = q.nth;
  auto r4 = [](int x) { return (x + 3) & ~3; };
  const int R = r4(ns), K = r4(nk);
  L.nspec = ns;
  L.nk = nk;
  L.nth = nth;
  L.nth_magic = static_cast<unsigned>(0x100000000ULL / static_cast<unsigned>(nth)) + 1u;
  int o = 0;
  L.pwsig = o; o += K;
  L.pwdir = o; o += K;
  L.tail = o; o += r4(7 * kJtot + 1);
  L.ec = o; o += r4(nth);
  L.es = o; o += r4(nth);
  L.common = o;
  // Per slot; offsets of slot 0, the others ws further on. SPEC rows start on 16 bytes, and ws is
  // 4 floats more than a multiple of 32, so four lanes reading float4s of four slots meet
  // different banks.
  L.spec = o; o += R;
  L.llws = o; o += r4((R + 3) / 4);
  L.wn1 = o; o += K;
  L.cg1 = o; o += K;
  L.dam = o; o += K;
  L.pwwn = o; o += K;
  L.mft = o; o += K;
  L.cbeta = o; o += K;
  L.wnf = o; o += K;
  L.dirf = o; o += r4(nth);
  L.jt = o; o += 4 * kJtot4;
  L.ws = o - L.common;
  while (L.ws % 32 != 4) L.ws += 4;
  L.tslot = 2 * R + r4((R + 3) / 4) + 8 * K;                  // closing sums + W3SPR4
  if (R + kNkWork * K > L.tslot) L.tslot = R + kNkWork * K;     // W3SDS4
  const int sin4 = 2 * R + r4((R + 3) / 4) + 8 * K;
  if (sin4 > L.tslot) L.tslot = sin4;
  const int seq = 3 * r4(nth) + 9 * K;
  if (seq > L.tslot) L.tslot = seq;
  while (L.tslot % 32 != 4) L.tslot += 4;
  L.alen = (n.nfrchg + 1) * nth;
  L.dia = r4((n.nfrhgh + 1) * nth) + 2 * r4(L.alen) + K;
  int g = 0;
  L.specinit = g; g += R;
  L.vdin = g; g += R;
  L.vsnl = g; g += R;
  L.vdnl = g; g += R;
  L.vsds = g; g += R;
  L.vdds = g; g += R;
  L.vsdb = g; g += R;
  // The DIA's DA1P DA1M DA2P DA2M and DA1C + DA2C; W3SDS4's two bin arrays (SSDSC(1) = 2, 3).
  L.da = g;
  const int d = 4 * r4(L.alen) + R;
  g += d > 2 * R ? d : 2 * R;
  L.total_g = (g + 31) & ~31;
  L.total_s = srce_shared_floats(L, 1);
  return L;
}

/// The named barriers of a CTA: its working warps' own, and the two over which they hand the tail to the
/// tail warp and take its results. They follow code in which lanes diverge, and nothing makes a warp's
/// lanes issue an inline assembly statement together (__syncwarp only makes them meet before it), so
/// these are PTX's barrier.sync and barrier.arrive, which do not ask for that; bar.sync and bar.arrive
/// are their .aligned forms, which do, and a warp that came apart could pass early or wait for good.
/// __syncwarp keeps the usual case one instruction for the warp.
constexpr int kBarWork = 1, kBarTail = 2, kBarTailDone = 3;
#if defined(__CUDACC__)
template <int ID>
__device__ __forceinline__ void barrier_sync(int threads) {
  __syncwarp();
  asm volatile("barrier.sync %0, %1;" ::"n"(ID), "r"(threads) : "memory");
}
template <int ID>
__device__ __forceinline__ void barrier_arrive(int threads) {
  __threadfence_block();
  __syncwarp();
  asm volatile("barrier.arrive %0, %1;" ::"n"(ID), "r"(threads) : "memory");
}
#endif

/// The working warps of a CTA (on the host: one warp of one lane).
struct Grp {
  int tid, nthr;
  WWB_PD void sync() const {
#if defined(__CUDA_ARCH__)
    barrier_sync<kBarWork>(nthr);
#endif
  }
  WWB_PD void syncwarp() const {
#if defined(__CUDA_ARCH__)
    __syncwarp();
#endif
  }
  /// All working warps announce to / wait for the tail warp.
  WWB_PD void tail_go() const {
#if defined(__CUDA_ARCH__)
    barrier_arrive<kBarTail>(nthr + 32);
#endif
  }
  WWB_PD void tail_wait() const {
#if defined(__CUDA_ARCH__)
    barrier_sync<kBarTailDone>(nthr + 32);
#endif
  }
#if defined(__CUDA_ARCH__)
  static constexpr int kLanes = 32;
  WWB_PD int warp() const { return tid >> 5; }
  WWB_PD int lane() const { return tid & 31; }
#else
  static constexpr int kLanes = 1;
  WWB_PD int warp() const { return 0; }
  WWB_PD int lane() const { return 0; }
#endif
  WWB_PD int nwarp() const { return (nthr + kLanes - 1) / kLanes; }
  /// Whether this warp runs the serial role r.
  WWB_PD bool role(int r) const { return warp() == r % nwarp(); }
};

/// In a loop's body: keeps the compiler from making a copy of the loop for each value of the flags that
/// do not change in it (it does not duplicate what the lanes of a warp agree on). The copies made the
/// kernel several times larger than the instruction cache.
WWB_PD void one_copy() {
#if defined(__CUDA_ARCH__)
  (void)__activemask();
#endif
}

/// Up to kSlots slot numbers, in registers.
struct SlotList {
  int n;
  unsigned ids;
  WWB_PD void add(int k) {
    ids |= static_cast<unsigned>(k) << (4 * n);
    ++n;
  }
  WWB_PD int at(int j) const { return (ids >> (4 * j)) & 15; }
  /// Entries j .. j + most - 1 of the list.
  WWB_PD SlotList part(int j, int most) const {
    return SlotList{n - j < most ? n - j : most, ids >> (4 * j)};
  }
};
static_assert(kSlots <= 8, "SlotList holds eight 4-bit numbers");
/// Slots that W3SDS4's sums over tables take together, so that a table row is read once for all of them
/// (9,520 points: two 106.7 ms, four 102.3, eight 106.8; 777 points with Romero's breaking: 19.1, 19.2, 20.4).
constexpr int kTogether = 4;

/// What the working warps leave for the tail warp.
struct TailBox {
  SlotList l;
  int exit;
};

/// What the CTA's phases read: the tables of one grid and the slots' memory. NTH: the number of
/// directions where the kernel is built for it (bin addresses and the loops over directions are then
/// compile-time arithmetic), 0 for any.
template <int NTH>
struct SrceGroup {
  const srce::Params* p;
  const SrceGrid* g;
  const st4::Params* q;
  const Fields* f;
  const Snl1Dev* n;
  const SrceLayout* L;
  float* w;    ///< shared
  float* gw;   ///< global scratch of the CTA
  float* t;    ///< the transient region
  SrceSh* sh;  ///< kSlots of them
  int ns;
  TailBox* box;  ///< null: the tail runs where it is called
  static constexpr int kNth = NTH;
  WWB_PD int nth() const { return NTH ? NTH : L->nth; }
  WWB_PD float* s(int k, int off) const { return w + off + k * L->ws; }
  WWB_PD float* gs(int k, int off) const { return gw + (off + k * L->total_g); }
  WWB_PD float* tr(int k) const { return t + k * L->tslot; }
  /// ECOS and ESIN of frequency ik: the one row kept in shared memory where every row of the registered
  /// arrays is the same, so that a chain does not wait for them.
  WWB_PD const float* ecos(int ik) const { return f->trig_rows ? w + L->ec : f->ecos + ik * nth(); }
  WWB_PD const float* esin(int ik) const { return f->trig_rows ? w + L->es : f->esin + ik * nth(); }
  WWB_PD unsigned char* llws(int k) const {
    return reinterpret_cast<unsigned char*>(w + L->llws + k * L->ws);
  }
  WWB_PD int row(int i) const {
    if (NTH) return static_cast<int>(static_cast<unsigned>(i) / (NTH ? NTH : 1));
#if defined(__CUDA_ARCH__)
    return static_cast<int>(__umulhi(static_cast<unsigned>(i), L->nth_magic));
#else
    return i / L->nth;
#endif
  }
};

/// f(setup(slot), i) for every bin i < n of the listed slots: a warp takes kLanes consecutive bins
/// of one slot at a time, slot after slot, so what setup returns (pointers, the point's scalars)
/// stays in registers. The chunks of all slots are dealt to the warps in one sequence.
template <class S, class F>
WWB_PD void bins(const Grp& c, const SlotList& l, int n, S setup, F f) {
  const int nw = c.nwarp(), nch = (n + Grp::kLanes - 1) / Grp::kLanes, turn = nch % nw;
  int first = c.warp();
WWB_UNROLL(1)
  for (int j = 0; j < l.n; ++j) {
    const auto s = setup(l.at(j));
WWB_UNROLL(1)
    for (int i = first * Grp::kLanes + c.lane(); i < n; i += nw * Grp::kLanes) {
      one_copy();
      f(s, i);
    }
    first -= turn;
    if (first < 0) first += nw;
  }
}
/// bins in two stages, U bins of a thread at a time: `ld` reads what a bin needs from global scratch,
/// `f` does the rest, so U bins' loads are in flight together. `end(s)` follows each slot.
template <int U, class S, class Ld, class F, class E>
WWB_PD void bins_ld(const Grp& c, const SlotList& l, int n, S setup, Ld ld, F f, E end) {
  const int nw = c.nwarp(), nch = (n + Grp::kLanes - 1) / Grp::kLanes, turn = nch % nw;
  const int step = nw * Grp::kLanes;
  int first = c.warp();
WWB_UNROLL(1)
  for (int j = 0; j < l.n; ++j) {
    auto s = setup(l.at(j));
WWB_UNROLL(1)
    for (int i = first * Grp::kLanes + c.lane(); i < n; i += U * step) {
      one_copy();
      decltype(ld(s, i)) in[U];
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
      for (int u = 0; u < U; ++u) in[u] = ld(s, i + u * step < n ? i + u * step : i);
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
      for (int u = 0; u < U; ++u)
        if (i + u * step < n) f(s, i + u * step, in[u]);
    }
    end(s);
    first -= turn;
    if (first < 0) first += nw;
  }
}
/// f(ith-setup, slot, row) for the nrow rows of every listed slot: a thread keeps its direction, so
/// what depends on the direction only is formed once.
template <class S, class F>
WWB_PD void dirs(const Grp& c, const SlotList& l, int nth, int nrow, S setup, F f) {
  const bool wide = c.nthr >= nth;
  const int g = wide ? c.nthr / nth : 1, r0 = wide ? c.tid / nth : 0;
  if (r0 >= g) return;
WWB_UNROLL(1)
  for (int ith = wide ? c.tid - r0 * nth : c.tid; ith < nth; ith += wide ? nth : c.nthr) {
    const auto s = setup(ith);
    int j = 0, r = r0;
    for (;;) {
      while (r >= nrow && j < l.n) {
        r -= nrow;
        ++j;
      }
      if (j >= l.n) break;
      one_copy();
      f(s, l.at(j), r);
      r += g;
    }
  }
}
/// f(slot, i) for every bin i < n of the listed slots.
template <class F>
WWB_PD void each_bin(const Grp& c, const SlotList& l, int n, F f) {
  bins(c, l, n, [](int k) { return k; }, [&](int k, int i) { f(k, i); });
}
/// f(slot, r) for r < n of the listed slots, one pair per thread.
template <class F>
WWB_PD void each_row(const Grp& c, const SlotList& l, int n, F f) {
WWB_UNROLL(1)
  for (int e = c.tid; e < l.n * n; e += c.nthr) {
    const int j = e / n;
    one_copy();
    f(l.at(j), e - j * n);
  }
}
/// f(slot) on warp r: lane k runs the k-th listed slot's chain.
template <class F>
WWB_PD void each_chain(const Grp& c, int r, const SlotList& l, F f) {
  if (!c.role(r)) return;
#if defined(__CUDA_ARCH__)
  if (c.lane() < l.n) f(l.at(c.lane()));
#else
  for (int j = 0; j < l.n; ++j) f(l.at(j));
#endif
}
/// f(r, slot) for nr chains of a kind on warp w, lane r * kSlots + j running chain r of the j-th listed
/// slot: one instruction serves all of them.
template <class F>
WWB_PD void each_chain_of(const Grp& c, int w, int nr, const SlotList& l, F f) {
  if (!c.role(w)) return;
#if defined(__CUDA_ARCH__)
  const int r = c.lane() / kSlots, j = c.lane() % kSlots;
  if (r < nr && j < l.n) f(r, l.at(j));
#else
  for (int r = 0; r < nr; ++r)
    for (int j = 0; j < l.n; ++j) f(r, l.at(j));
#endif
}

struct F4 {
  float a, b, c, d;
};
/// Four floats from 16-byte aligned memory.
WWB_PD F4 ld4(const float* p) {
#if defined(__CUDA_ARCH__)
  const float4 v = *reinterpret_cast<const float4*>(p);
  return F4{v.x, v.y, v.z, v.w};
#else
  return F4{p[0], p[1], p[2], p[3]};
#endif
}
/// f(x[i], i) for i = 0 .. n - 1 in order, x 16-byte aligned: one load per four values.
template <class F>
WWB_PD void walk4(const float* x, int n, F f) {
  int i = 0;
WWB_UNROLL(4)
  for (; i + 4 <= n; i += 4) {
    const F4 v = ld4(x + i);
    f(v.a, i);
    f(v.b, i + 1);
    f(v.c, i + 2);
    f(v.d, i + 3);
  }
WWB_UNROLL(1)
  for (; i < n; ++i) f(x[i], i);
}
/// The sum of x[0 .. n) in order from v.
WWB_PD float sum4(const float* x, int n, float v) {
  walk4(x, n, [&](float a, int) { v = v + a; });
  return v;
}
/// The sum of the nth values of row ik of a bin array that starts on 16 bytes.
WWB_PD float row_sum(const float* x, int ik, int nth) {
  const float* const r = x + ik * nth;
  float v = 0.0f;
  if ((nth & 3) == 0) return sum4(r, nth, v);
WWB_UNROLL(1)
  for (int j = 0; j < nth; ++j) v = v + r[j];
  return v;
}

/// The sum of the terms whose flag is `want`, in order from v, terms and flags 16- and 4-byte aligned.
/// The others add -0, which changes no sum: a branch per term would diverge between the slots.
WWB_PD float sum_flagged(const float* x, const unsigned char* flag, int n, unsigned want, float v) {
  int i = 0;
WWB_UNROLL(4)
  for (; i + 4 <= n; i += 4) {
    const F4 q = ld4(x + i);
    const uint32_t b = *reinterpret_cast<const uint32_t*>(flag + i);
    v = v + ((b & 0xffu) == want ? q.a : -0.0f);
    v = v + ((b >> 8 & 0xffu) == want ? q.b : -0.0f);
    v = v + ((b >> 16 & 0xffu) == want ? q.c : -0.0f);
    v = v + ((b >> 24) == want ? q.d : -0.0f);
  }
WWB_UNROLL(1)
  for (; i < n; ++i) v = v + (flag[i] == want ? x[i] : -0.0f);
  return v;
}

/// The same for n known when compiled and a multiple of 4: all loads first.
template <int N>
WWB_PD float sum_flagged_n(const float* x, const unsigned char* flag, unsigned want, float v) {
  F4 q[N / 4];
  uint32_t b[N / 4];
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
  for (int i = 0; i < N / 4; ++i) {
    q[i] = ld4(x + 4 * i);
    b[i] = *reinterpret_cast<const uint32_t*>(flag + 4 * i);
  }
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
  for (int i = 0; i < N / 4; ++i) {
    v = v + ((b[i] & 0xffu) == want ? q[i].a : -0.0f);
    v = v + ((b[i] >> 8 & 0xffu) == want ? q[i].b : -0.0f);
    v = v + ((b[i] >> 16 & 0xffu) == want ? q[i].c : -0.0f);
    v = v + ((b[i] >> 24) == want ? q[i].d : -0.0f);
  }
  return v;
}

WWB_PD float powf_i(float x, float y) { return dm::powf_t<WWB_POWF_FUSE>(x, y); }
/// Sine and cosine without a call: its results would pass through memory.
WWB_PD void sincosf_i(float x, float* s, float* c) { dm::sincosf_t<WWB_SINCOSF_FUSE>(x, s, c); }

// ------------------------------------------------------------------ what the slots share
/// The powers of SIG that W3SPR4 takes and the analytic tail's terms that depend on J only
/// (:886-917 of W3SIN4): functions of the grid, formed once per CTA.
template <class G>
WWB_PD void srce_common(const Grp& c, const G& x) {
  const SrceLayout& L = *x.L;
  const st4::Params& q = *x.q;
  const Fields& f = *x.f;
  if (f.trig_rows) {
WWB_UNROLL(1)
    for (int i = c.tid; i < x.nth(); i += c.nthr) {
      x.w[L.ec + i] = f.ecos[i];
      x.w[L.es + i] = f.esin[i];
    }
  }
WWB_UNROLL(1)
  for (int ik = c.tid; ik < L.nk; ik += c.nthr) {
    x.w[L.pwsig + ik] = dm::powf(f.sig[ik + 1], 2.0f * q.wwnmeanptail);
    x.w[L.pwdir + ik] = dm::powf(f.sig[ik + 1], q.ssdsc[11]);
  }
  if (q.sintailpar[0] < 0.5f) {
    float* const t = x.w + L.tail;
    const float signk = f.sig[L.nk];
    const float zinf = dm::logf(signk * signk / kGrav);
    const float dely = (kLogTpiOver005 - zinf) / static_cast<float>(kJtot);
WWB_UNROLL(1)
    for (int j = c.tid; j < kJtot; j += c.nthr) {
      const float y = dm::expf(zinf + static_cast<float>(j) * dely);
      const float ykm = (y / kKm);
      const float ykm2 = ykm * ykm;
      const float tensk = 1.0f + ykm2;
      const float cm = sqrt_f(kGrav * tensk / y);
      t[j] = cm;
      t[kJtot + j] = 0.5f * (3.0f * ykm2 + 1.0f) * sqrt_f(kGrav / (y * tensk));
      t[4 * kJtot + j] = cm * cm;
      // 0 where div_by's two steps might not be exact
      t[6 * kJtot + j] = cm >= 0x1p-20f && cm <= 0x1p20f ? 1.0f / cm : 0.0f;
      if (j == 0) t[7 * kJtot] = dely;
      t[5 * kJtot + j] = kCmm / cm;
      if (q.sintailpar[2] > 0.0f) {
        const float ykm1 = (ykm - 1.0f);
        t[2 * kJtot + j] = dm::expf(-0.25f * (ykm1 * ykm1));
        t[3 * kJtot + j] = dm::tanhf((y - 20.0f) / 5.0f);
      }
    }
  }
  c.sync();
}

// ------------------------------------------------------------------ W3SRCE's initialisation
/// The start of section 1 (:869-1073) for points just loaded: spec, wn1, cg1 and the packets are
/// in the slots; the slots' state is set.
template <class G>
WWB_PD void srce_begin(const Grp& c, const G& x, const SlotList& l) {
  const srce::Params& p = *x.p;
  const SrceLayout& L = *x.L;
  each_bin(c, l, L.nspec, [&](int k, int i) {
    // LLWS is 1 at IT = 0 (:1073); otherwise the reference reads it unset at :1080, where only
    // FMEANWS depends on it and :1119 overwrites that: start from 0.
    x.llws(k)[i] = x.sh[k].in.it == 0 ? 1 : 0;
    x.gs(k, L.vsdb)[i] = 0.0f;
  });
  each_row(c, l, L.nk, [&](int k, int ik) {
    const float w = x.s(k, L.wn1)[ik];
    x.s(k, L.dam)[ik] = p.facp / (x.g->sig[ik] * (w * (w * w)));
    x.s(k, L.pwwn)[ik] = dm::powf(w, x.q->wwnmeanp);
    {
      // W3SBT1's factor (:1339): K, CG, SIG and the depth only.
      const float factor = p.sbtc1 / mx(x.sh[k].in.d_inp, p.dmin);
      const float xx = x.s(k, L.cg1)[ik] * w / x.g->sig[ik] - 0.5f;
      x.s(k, L.cbeta)[ik] = factor * (xx > 0.0f ? xx : 0.0f);
    }
    if (x.sh[k].in.flogrd58) {
      // W3SDS4's mean foam thickness (:2604-2628) depends on K and SIG only.
      const float sig = x.f->sig[ik + 1];
      const float tstr = kTstrFac / sig;
      const float tmax = kTmaxFac / sig;
      const float dt = tmax / 50.0f;
      float mft = 0.0f;
WWB_UNROLL(1)
      for (int it = 1; it <= 50; ++it) {
        const float t = static_cast<float>(it) * dt;
        if (t < tstr) {
          mft = mft + ((0.4f / (w * tstr)) * t) * dt;
        } else {
          mft = mft + ((0.4f / w) * dm::expf(-((t - tstr) / 3.8f))) * dt;
        }
      }
      x.s(k, L.mft)[ik] = mft / tmax;
    }
  });
  each_chain(c, 1, l, [&](int k) {
    // W3SBT1's cut: bins from the first frequency with K * DEPTH > 6 on have no friction; all of
    // them when that is the first one.
    const float depth = mx(x.sh[k].in.d_inp, p.dmin);
    const float* const wn = x.s(k, L.wn1);
    int ik = 0;
WWB_UNROLL(1)
    for (; ik < L.nk; ++ik)
      if (wn[ik] * depth > 6.0f) break;
    x.sh[k].nscut = ik == 0 ? -1 : ik * x.nth();
  });
  each_chain(c, 0, l, [&](int k) {
    SrceSh& s = x.sh[k];
    const SrceIn& in = s.in;
    s.depth = mx(in.d_inp, p.dmin);
    s.drat = in.dair / kDwat;
    s.icescaleln = mx(mn(1.0f - in.ice * p.icescales[0], 1.0f), 0.0f);
    s.icescalein = mx(mn(1.0f - in.ice * p.icescales[1], 1.0f), 0.0f);
    s.icescalenl = mx(mn(1.0f - in.ice * p.icescales[2], 1.0f), 0.0f);
    s.icescaleds = mx(0.0f, mn(1.0f - in.ice * p.icescales[3], 1.0f));
    s.dtdyn = 0.0f;
    s.dttot = 0.0f;
    s.nsteps = 0;
    s.phiaw = 0.0f;
    s.r.charn = 0.0f;
    s.tws = 0.0f;
    s.phibbl = 0.0f;
    s.tauwix = s.tauwiy = s.tauwnx = s.tauwny = 0.0f;
    s.tauwax = s.tauway = 0.0f;
    s.taubbl[0] = s.taubbl[1] = s.tauice[0] = s.tauice[1] = 0.0f;
    s.phice = s.tauocx = s.tauocy = 0.0f;
    s.r.wnmean = 0.0f;
    s.r.dlwmean = 0.0f;
    s.vddb = 0.0f;
    for (int j = 0; j < 4; ++j) s.whitecap[j] = 0.0f;
    if (x.q->sintailpar[3] > 0.5f) {
      s.tauwx = 0.0f;
      s.tauwy = 0.0f;
    }
    if (in.it == 0) {
      s.tauwx = s.tauwy = 0.0f;
      s.r.ustar = 0.0f;
      s.r.usdir = 0.0f;
    }
    float sn, cs;
    dm::sincosf(in.u10dir, &sn, &cs);
    s.sinw = sn;
    s.cosw = cs;
    {
      const float signk = x.f->sig[L.nk];
      const float s2 = signk * signk;
      const float s5 = s2 * (s2 * signk);
      s.c0 = x.q->dth * s5 / kGrav2Tpi * kTpi * signk / x.s(k, L.cg1)[L.nk - 1];
    }
  });
  c.sync();
}

// ------------------------------------------------------------------------------------ W3SPR4
/// W3SPR4 (w3src4md.F90:142-384) of the listed slots, first phase: the per-IK direction sums and
/// the terms of the moments (:245-300); the arrays T0 .. T5 and SIGFAC stay in the slot's transient
/// region from `off` on. The libmvec powers of :316 and :317 use scalar powf in every lane; the
/// powers are functions of the grid or of the point's WN and are kept (x.w pwsig, pwdir, pwwn).
template <class G>
WWB_PD void spr4_sums(const Grp& c, const G& x, const SlotList& l, int off) {
  const SrceLayout& L = *x.L;
  const Fields& f = *x.f;
  const int nk = L.nk, nth = x.nth();
  each_row(c, l, nk, [&](int k, int ik) {
    const float* const a = x.s(k, L.spec) + ik * nth;
    const unsigned char* const lw = x.llws(k) + ik * nth;
    float ebk = 0.0f, eb2k = 0.0f;
    if ((nth & 3) == 0) {
WWB_UNROLL(1)
      for (int i = 0; i < nth; i += 4) {
        const F4 v = ld4(a + i);
        const uint32_t b = *reinterpret_cast<const uint32_t*>(lw + i);
        ebk = ebk + v.a;
        if (b & 0xffu) eb2k = eb2k + v.a;
        ebk = ebk + v.b;
        if (b & 0xff00u) eb2k = eb2k + v.b;
        ebk = ebk + v.c;
        if (b & 0xff0000u) eb2k = eb2k + v.c;
        ebk = ebk + v.d;
        if (b & 0xff000000u) eb2k = eb2k + v.d;
      }
    } else {
WWB_UNROLL(1)
      for (int i = 0; i < nth; ++i) {
        ebk = ebk + a[i];
        if (lw[i] != 0) eb2k = eb2k + a[i];
      }
    }
    const float dden = f.dden[ik], cg = x.s(k, L.cg1)[ik];
    const float b = ebk * dden / cg;
    const float b2 = eb2k * dden / cg;
    float* const t = x.tr(k) + off + ik;
    t[0] = b;
    t[nk] = b / f.sig[ik + 1];
    t[2 * nk] = b * x.w[L.pwsig + ik];
    t[3 * nk] = b * x.s(k, L.pwwn)[ik];
    t[4 * nk] = b2;
    t[5 * nk] = b2 * x.w[L.pwsig + ik];
    t[6 * nk] = x.w[L.pwdir + ik] * dden / cg;
  });
}

/// Second phase, roles 0-3: the moments with CALC_USTAR, and the running sums ELCS, ELSN and the
/// running MAX over all bins. Each chain is 5 k cycles at 36 x 36 and the moments 15 k (ten Newton
/// steps of CALC_USTAR); side by side they cost the longest one.
template <class G>
WWB_PD void spr4_chains(const Grp& c, const G& x, const SlotList& l, int off) {
  const SrceLayout& L = *x.L;
  const st4::Params& p = *x.q;
  const Fields& f = *x.f;
  const int nk = L.nk, nth = x.nth();
  each_chain(c, 0, l, [&](int k) {
    SrceSh& s = x.sh[k];
    const float* const t = x.tr(k) + off;
    const float eps = 1.E-7f;
    float ustar = max_r(0.0001f, s.r.ustar);
    float emean = 0.0f, fmean = 0.0f, fmean1 = 0.0f, wnmean = 0.0f, emeanws = 0.0f,
          fmeanws = 0.0f;
WWB_UNROLL(4)
    for (int ik = 0; ik < nk; ++ik) {
      emean = emean + t[ik];
      fmean = fmean + t[nk + ik];
      fmean1 = fmean1 + t[2 * nk + ik];
      wnmean = wnmean + t[3 * nk + ik];
      emeanws = emeanws + t[4 * nk + ik];
      fmeanws = fmeanws + t[5 * nk + ik];
    }
    float eband = t[nk - 1] / f.dden[nk - 1];
    emean = emean + eband * p.fte;
    fmean = fmean + eband * p.ftf;
    fmean1 = fmean1 + eband * p.sstxftftail;
    wnmean = wnmean + eband * p.sstxftwn;
    eband = t[5 * nk - 1] / f.dden[nk - 1];
    emeanws = emeanws + eband * p.fte;
    fmeanws = fmeanws + eband * p.sstxftftail;
    fmean = kTpiInv * emean / max_r(eps, fmean);
    if (fmean1 < eps) {
      fmean1 = kTpiInv * f.sig[nk];
    } else {
      fmean1 = kTpiInv * dm::powf(max_r(eps, fmean1) / max_r(eps, emean),
                                  1.0f / (2.0f * p.wwnmeanptail));
    }
    wnmean = dm::powf(max_r(eps, wnmean) / max_r(eps, emean), 1.0f / p.wwnmeanp);
    if (fmeanws < eps || emeanws < eps) {
      fmeanws = kTpiInv * f.sig[nk];
    } else {
      fmeanws = kTpiInv * dm::powf(max_r(eps, fmeanws) / max_r(eps, emeanws),
                                   1.0f / (2.0f * p.wwnmeanptail));
    }
    const float u = s.in.u10abs;
    const float tauw = sqrt_f(s.tauwx * s.tauwx + s.tauwy * s.tauwy);
    float z0 = s.r.z0, charn = s.r.charn;
    calc_ustar(p, f, u, tauw, &ustar, &z0, &charn);
    const float unz = max_r(0.01f, u);
    const float r = ustar / unz;
    s.r.ustar = ustar;
    s.r.usdir = s.in.u10dir;
    s.r.emean = emean;
    s.r.fmean = fmean;
    s.r.fmean1 = fmean1;
    s.r.wnmean = wnmean;
    s.r.cd = r * r;
    s.r.z0 = z0;
    s.r.charn = charn;
    s.r.fmeanws = fmeanws;
  });
WWB_UNROLL(1)
  each_chain_of(c, 1, 2, l, [&](int comp, int k) {
      const float* const a = x.s(k, L.spec);
      const float* const sf = x.tr(k) + off + 6 * nk;
        float v = 0.0f;
WWB_UNROLL(1)
      for (int ik = 0; ik < nk; ++ik) {
        const float sfk = sf[ik];
        const float* const ar = a + ik * nth;
        const float* const er = comp ? x.esin(ik) : x.ecos(ik);
        int i = 0;
        if ((nth & 3) == 0) {
WWB_UNROLL(3)
          for (; i < nth; i += 4) {
            const F4 q = ld4(ar + i), r = ld4(er + i);
            v = v + q.a * r.a * sfk;
            v = v + q.b * r.b * sfk;
            v = v + q.c * r.c * sfk;
            v = v + q.d * r.d * sfk;
          }
        }
WWB_UNROLL(1)
        for (; i < nth; ++i) v = v + ar[i] * er[i] * sfk;
      }
      x.sh[k].chains[comp] = v;
    });
  each_chain(c, 3, l, [&](int k) {
    float v = 0.0f;
    walk4(x.s(k, L.spec), L.nspec, [&](float a, int) { v = max_r(v, a); });
    x.sh[k].chains[2] = v;
  });
}

// ------------------------------------------------------------------------------------ W3SIN4
/// What one direction of the stress scan needs from its frequency and its point.
struct ScanK {
  float cm, ucn, const2, cnst, zcn, swv, swt, sig2is;
};
/// The swell damping's scalars of a point.
struct Swell {
  float fwuorb, fu, fud, pturb, pvisc;
};
/// DSTAB and LLWS of one bin (:739-783).
WWB_PD float scan_bin(const st4::Params& p, const Swell& s, const ScanK& q, float ustar, float ustp,
                      float coswind, int* lw) {
  float dst = 0.0f;
  int l = 0;
  if (coswind > 0.01f) {
    const float zarg = kKappa / (coswind * q.ucn);
    const float zlog = q.zcn + zarg;
    if (zlog < 0.0f) {
      const float zlog2 = zlog * zlog;
      dst = q.cnst * dm::expf(zlog) * (zlog2 * zlog2) * q.ucn * q.ucn * dm::powf(coswind, p.ssinthp);
      l = 1;
    }
    if (28.0f * q.cm * ustar * coswind >= 1.0f) l = 1;
  }
  *lw = l;
  if ((p.sswellf[0] != 0.0f && dst < 1E-7f * q.sig2is) || p.sswellf[2] > 0.0f) {
    const float dvisc = q.swv;
    const float dturb = q.swt * (s.fwuorb + (s.fu + s.fud * coswind) * ustp);
    dst = dst + s.pturb * dturb + s.pvisc * dvisc;
  }
  return dst;
}
/// The same without a branch, so that the bins of a thread overlap: 0 < SSINTHP < 16 (a cosine between
/// 0.01 and 1 to that power has no special case); *ok is cleared where the division is not div_core's.
WWB_PD float scan_bin_q(const st4::Params& p, const Swell& s, const ScanK& q, float ustar, float ustp,
                        float coswind, int* lw, bool* ok) {
  const bool up = coswind > 0.01f;
  const float xx = up ? coswind * q.ucn : 1.0f;
  *ok = *ok && dm::div_ok(kKappa, xx);
  const float zlog = q.zcn + dm::div_core(kKappa, xx);
  const bool grow = up && zlog < 0.0f;
  const float zl = grow ? zlog : -1.0f, cw = grow ? coswind : 0.5f;
  const float zlog2 = zl * zl;
  const float g = q.cnst * dm::expf_neg(zl) * (zlog2 * zlog2) * q.ucn * q.ucn *
                  dm::powf_mid(cw, p.ssinthp);
  float dst = grow ? g : 0.0f;
  *lw = grow || (up && 28.0f * q.cm * ustar * coswind >= 1.0f) ? 1 : 0;
  const float dturb = q.swt * (s.fwuorb + (s.fu + s.fud * coswind) * ustp);
  const float damped = dst + s.pturb * dturb + s.pvisc * q.swv;
  return (p.sswellf[0] != 0.0f && dst < 1E-7f * q.sig2is) || p.sswellf[2] > 0.0f ? damped : dst;
}
WWB_PD bool scan_plain(const st4::Params& p) { return p.ssinthp > 0.0f && p.ssinthp < 16.0f; }

/// Offsets of W3SIN4's NK arrays in a slot's transient region (after the 2 R + R/4 floats of the
/// stress terms and their signs).
struct Sin4At {
  int zcn, cm, const2, cnst, swv, swt, tu, ta;
};
/// The tail's arrays in a slot's L.jt.
enum TailAt : int { kGz = 0, kZb = kJtot4, kUs = 2 * kJtot4, kLev = 3 * kJtot4 };
WWB_PD Sin4At sin4_at(const SrceLayout& L) {
  const int R = (L.nspec + 3) & ~3, K = (L.nk + 3) & ~3;
  const int o = 2 * R + ((((R + 3) / 4) + 3) & ~3);
  return Sin4At{o, o + K, o + 2 * K, o + 3 * K, o + 4 * K, o + 5 * K, o + 6 * K, o + 7 * K};
}

template <class G>
WWB_PD ScanK scan_k(const G& x, const Sin4At& at, const float* tr, int ik, float ustp) {
  const float* const t = tr + ik;
  ScanK q;
  q.cm = t[at.cm];
  q.ucn = ustp * q.cm + x.q->zzalp;
  q.const2 = t[at.const2];
  q.cnst = t[at.cnst];
  q.zcn = t[at.zcn];
  q.swv = t[at.swv];
  q.swt = t[at.swt];
  q.sig2is = x.f->sig2[ik * x.nth()];
  return q;
}

/// Lanes that share one point's stress scan: 36 directions in three rounds, 24 in two; two points
/// to a warp (18 lanes and one point: no faster at 36 directions, 6 % slower at 24).
#if defined(__CUDA_ARCH__)
constexpr int kScanLanes = 12;
#else
constexpr int kScanLanes = 1;
#endif

/// The stress scan over IK (:696-797) for slots whose running stress feeds the next frequency
/// (TTAUWSHELTER /= 0) or that the parallel form leaves to it. A team of kScanLanes lanes takes one
/// point: every lane forms the frequency's scalars, the directions are split, and the four ordered
/// sums (x and y, by the sign of DSTAB) are one lane each.
template <class G>
WWB_PD void scan_serial(const Grp& c, const G& x, const SlotList& l, const Sin4At& at) {
  const SrceLayout& L = *x.L;
  const st4::Params& p = *x.q;
  const int nk = L.nk, nth = x.nth(), T4 = (nth + 3) & ~3;
  const bool plain = scan_plain(p);
  constexpr int kPerWarp = Grp::kLanes / kScanLanes;
  const int team = c.lane() / kScanLanes, sub = c.lane() - team * kScanLanes;
WWB_UNROLL(1)
  for (int j0 = c.warp() * kPerWarp; j0 < l.n; j0 += c.nwarp() * kPerWarp) {
    const int j = j0 + team;
    const bool on = team < kPerWarp && j < l.n;
    const int k = l.at(on ? j : j0);
    SrceSh& s = x.sh[k];
    float* const t = x.tr(k);
    float* const bx = t;
    float* const by = t + T4;
    unsigned char* const neg = reinterpret_cast<unsigned char*>(t + 2 * T4);
    const float* const a = x.s(k, L.spec);
    unsigned char* const llws = x.llws(k);
    float* const vdin = x.gs(k, L.vdin);
    const Swell sw{s.fwuorb, s.fu, s.fud, s.pturb, s.pvisc};
    const float ustar = s.r.ustar, shelter = fabs_f(p.ttauwshelter);
    float ust = ustar, taux = 0.0f, tauy = 0.0f, cosu = 0.0f, sinu = 0.0f, ustp = 0.0f;
    const int first = p.stab3 ? 1 : 3, last = p.stab3 ? 2 : 3;
WWB_UNROLL(1)
    for (int istab = first; istab <= last; ++istab) {
      if (istab == 1) ust = ustar * (1.0f - s.ustarsigma);
      if (istab == 2) ust = ustar * (1.0f + s.ustarsigma);
      taux = (ust * ust) * s.cosw;
      tauy = (ust * ust) * s.sinw;
      if (on)
WWB_UNROLL(1)
        for (int q = sub; q < 4; q += kScanLanes) s.sums[q] = 0.0f;
      c.syncwarp();
WWB_UNROLL(1)
      for (int ik = 0; ik < nk; ++ik) {
        if (on) {
          const ScanK q0 = scan_k(x, at, t, ik, 0.0f);  // UCN needs USTP, below
          const float taupx = taux - shelter * s.sums[0];
          const float taupy = tauy - shelter * s.sums[1];
          const float tau2 = taupx * taupx + taupy * taupy;
          float root;
          bool bad = true;
          if (dm::normal_pos(tau2) && dm::atan2f_ok(taupy, taupx)) {
            // One block, so the power and the angle overlap.
            root = dm::powf_core(tau2, 0.25f);
            dm::sincosf_core(dm::atan2f_core(taupy, taupx, &bad), &sinu, &cosu);
          }
          if (bad) {
            root = dm::powf(tau2, 0.25f);
            dm::sincosf(dm::atan2f(taupy, taupx), &sinu, &cosu);
          }
          ustp = min_r(root, max_r(ust, 0.3f));
          ScanK q = q0;
          q.ucn = ustp * q.cm + p.zzalp;
          // Rounds of kRound directions a lane, each a block without branches.
          constexpr int kRound = G::kNth != 0 && G::kNth % kScanLanes == 0 && G::kNth / kScanLanes <= 4
                                     ? G::kNth / kScanLanes : 1;
WWB_UNROLL(1)
          for (int ith = sub; ith < nth; ith += kRound * kScanLanes) {
            one_copy();
            float dst[kRound], cw[kRound], ec[kRound], es[kRound];
            int lw[kRound];
            bool ok = plain;
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
            for (int r = 0; r < kRound; ++r) {
              const int d = ith + r * kScanLanes;
              ec[r] = x.ecos(ik)[d];
              es[r] = x.esin(ik)[d];
              cw[r] = (ec[r] * cosu + es[r] * sinu);
              dst[r] = scan_bin_q(p, sw, q, ustar, ustp, cw[r], &lw[r], &ok);
            }
            if (!ok) {
WWB_UNROLL(1)
              for (int r = 0; r < kRound; ++r) dst[r] = scan_bin(p, sw, q, ustar, ustp, cw[r], &lw[r]);
            }
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
            for (int r = 0; r < kRound; ++r) {
              const int d = ith + r * kScanLanes, i = ik * nth + d;
              const float temp2 = q.const2 * dst[r] * a[i];
              bx[d] = temp2 * ec[r];
              by[d] = temp2 * es[r];
              neg[d] = dst[r] < 0.0f ? 1 : 0;
              vdin[i] = istab == 2 ? 0.5f * (vdin[i] + dst[r]) : dst[r];
              llws[i] = static_cast<unsigned char>(lw[r]);
            }
          }
        }
        c.syncwarp();
        if (on)
WWB_UNROLL(1)
          for (int q = sub; q < 4; q += kScanLanes) {
            const float* const b = (q & 1) ? by : bx;
            const unsigned want = static_cast<unsigned>(q >> 1);
            s.sums[q] = G::kNth != 0 && G::kNth % 4 == 0
                            ? sum_flagged_n<(G::kNth != 0 ? G::kNth : 4)>(b, neg, want, s.sums[q])
                            : sum_flagged(b, neg, nth, want, s.sums[q]);
          }
        c.syncwarp();
      }
      if (on && sub == 0) {
        s.ss[istab - 1][0] = s.sums[0];
        s.ss[istab - 1][1] = s.sums[1];
        s.sn[istab - 1][0] = s.sums[2];
        s.sn[istab - 1][1] = s.sums[3];
      }
      c.syncwarp();
    }
    if (on && sub == 0) {
      s.ust = ust;
      s.taux = taux;
      s.tauy = tauy;
      s.cosu = cosu;
      s.sinu = sinu;
      s.ustp = ustp;
    }
  }
}

/// a / b for b in [2^-20, 2^20], correctly rounded, from y = 1 / b correctly rounded (0: unknown): two steps q + (a - b q) y with fused
/// multiply-adds (Markstein 1990, IBM J. Res. Dev. 34: one step from a quotient within an ulp is exact,
/// the first makes it so), where nothing under- or overflows; else the division itself. The tail divides
/// by the same 50 phase speeds in every substep, and this is a third of a division's latency. a = -0 gives
/// +0, which changes no result there.
WWB_PD float div_by(float a, float b, float y) {
  const float m = fabs_f(a);
  if (!(((m >= 0x1p-80f && m <= 0x1p80f) || a == 0.0f) && y != 0.0f)) return a / b;
  float q = a * y;
  q = dm::fma_f(dm::fma_f(-b, q, a), y, q);
  return dm::fma_f(dm::fma_f(-b, q, a), y, q);
}

/// The serial part of W3SIN4's closing section for one slot (:799-955): the stresses, the tail's level
/// and the tail's recurrence (per step ZBETA and USTR**2 are kept, TAU1 is summed afterwards), or the
/// tabulated tail. 50 dependent steps of an exponential, a logarithm, a division and a square root: the
/// longest chain of a substep, so what does not depend on the step before is taken out of it.
template <class G>
WWB_PD void sin4_tail(const G& x, int k) {
  const SrceLayout& L = *x.L;
  const st4::Params& p = *x.q;
  const Fields& f = *x.f;
  const int nk = L.nk, nth = x.nth();
  SrceSh& s = x.sh[k];
  const float* const a = x.s(k, L.spec) + (nk - 1) * nth;
  float xstress, ystress, twnx, twny;
  if (!p.stab3) {
    xstress = s.ss[2][0];
    ystress = s.ss[2][1];
    twnx = s.sn[2][0];
    twny = s.sn[2][1];
  } else {
    xstress = 0.5f * (s.ss[0][0] + s.ss[1][0]);
    ystress = 0.5f * (s.ss[0][1] + s.ss[1][1]);
    twnx = 0.5f * (s.sn[0][0] + s.sn[1][0]);
    twny = 0.5f * (s.sn[0][1] + s.sn[1][1]);
  }
  s.tauwax = twnx;
  s.tauway = twny;
  s.stress[0] = xstress;
  s.stress[1] = ystress;
  float ustl;
  {
    const float taupx = s.taux - fabs_f(p.ttauwshelter) * xstress;
    const float taupy = s.tauy - fabs_f(p.ttauwshelter) * ystress;
    ustl = dm::powf((taupx * taupx + taupy * taupy), 0.25f);
    s.usdirpl = dm::atan2f(taupy, taupx);
  }
  const float ust3 = ustl, z0 = s.r.z0;
  float temp = 0.0f;
  {
    const float cosu = s.cosu, sinu = s.sinu;
    const float *const ec = x.ecos(nk - 1), *const es = x.esin(nk - 1);
WWB_UNROLL(6)
    for (int i = 0; i < nth; ++i) {
      const float coswind = (ec[i] * cosu + es[i] * sinu);
      const float cp = (max_r(coswind, 0.0f));
      temp = temp + a[i] * (cp * (cp * cp));
    }
  }
  const float levtail0 = s.c0 * temp;
  s.levtail0 = levtail0;
  if (p.sintailpar[0] < 0.5f) {
    const float* const tt = x.w + L.tail;
    float* const tr = x.s(k, L.jt);
    float ustr = ust3;
    const float dely = tt[7 * kJtot];
    float taur = ust3 * ust3;
    const float const1 = s.const1, zzalp = p.zzalp, sp1 = p.sintailpar[1];
    const bool lev = p.sintailpar[2] > 0.0f;
WWB_UNROLL(1)
    for (int j = 0; j < kJtot; ++j) {
      one_copy();
      const float cm = tt[j], cgtail = tt[kJtot + j], rcm = tt[6 * kJtot + j];
      const float zx = div_by(ustr, cm, rcm) + zzalp;
      const float zarg = min_r(kKappa / zx, 20.0f);
      const float zmu = min_r(tr[kGz + j] * dm::expf_q(zarg), 1.0f);
      const float zlog = min_r(dm::logf_q(zmu), 0.0f);
      const float zlog2 = zlog * zlog;
      const float zbeta = const1 * zmu * (zlog2 * zlog2);
      float levtail = levtail0;
      if (lev) {
        float alpham;
        if (ustr < cm) {
          alpham = max_r(0.0f, 0.01f * (1.0f + dm::logf(ustr / cm)));
        } else {
          alpham = 0.01f * (1.0f + 3.0f * dm::logf(ustr / cm));
        }
        const float fm = tt[2 * kJtot + j];
        const float alphat = alpham * tt[5 * kJtot + j] * fm;
        const float th = tt[3 * kJtot + j];
        levtail = levtail0 * 0.5f * (1.0f - th) + p.sintailpar[2] * 0.5f * (1.0f + th) * alphat;
        tr[kLev + j] = levtail;
      }
      const float us2 = ustr * ustr, w = (j == 0 || j == kJtot - 1) ? 0.5f : 1.0f;
      tr[kZb + j] = zbeta;
      tr[kUs + j] = us2;
      taur = taur - div_by(w * sp1 * us2 * zbeta * levtail * dely * cgtail, cm, rcm);
      ustr = sqrt_f(max_r(taur, 0.0f));
    }
  } else {
    const float xi = ust3 / p.delust;
    const int ind = max_i(1, min_i(st4::kIustar - 1, fint(xi)));
    const float deli1 = max_r(min_r(1.0f, xi - static_cast<float>(ind)), 0.0f);
    const float deli2 = 1.0f - deli1;
    const float ustm = max_r(ust3, 0.00001f);
    const float xj = max_r(0.0f, (kGrav * z0 / (ustm * ustm) - p.aalpha) / p.delalp);
    const int j = max_i(1, min_i(st4::kIalpha - 1, fint(xj)));
    const float delj1 = max_r(0.0f, min_r(1.0f, xj - static_cast<float>(j)));
    const float delj2 = 1.0f - delj1;
    float tau1;
    if (p.ttauwshelter > 0.0f) {
      const float xk = levtail0 / p.deltail;
      const int i = min_i(st4::kIlevTail - 1, fint(xk));
      const float delk1 = min_r(1.0f, xk - static_cast<float>(i));
      const float delk2 = 1.0f - delk1;
      tau1 = ((f.tauhft2_at(ind, j, i) * deli2 + f.tauhft2_at(ind + 1, j, i) * deli1) * delj2 +
              (f.tauhft2_at(ind, j + 1, i) * deli2 + f.tauhft2_at(ind + 1, j + 1, i) * deli1) *
                  delj1) * delk2 +
             ((f.tauhft2_at(ind, j, i + 1) * deli2 + f.tauhft2_at(ind + 1, j, i + 1) * deli1) *
                  delj2 +
              (f.tauhft2_at(ind, j + 1, i + 1) * deli2 +
               f.tauhft2_at(ind + 1, j + 1, i + 1) * deli1) *
                  delj1) *
                 delk1;
    } else {
      tau1 = (f.tauhft_at(ind, j) * deli2 + f.tauhft_at(ind + 1, j) * deli1) * delj2 +
             (f.tauhft_at(ind, j + 1) * deli2 + f.tauhft_at(ind + 1, j + 1) * deli1) * delj1;
    }
    s.tauhf = levtail0 * (ust3 * ust3) * tau1;
  }
}

/// 3. The tail stress and the stress limit (:799-976) of the listed slots, by one warp: TAUWX and TAUWY.
template <class G, class Sync>
WWB_PD void sin4_close(int lane, const G& x, const SlotList& l, Sync syncwarp) {
  const SrceLayout& L = *x.L;
  const st4::Params& p = *x.q;
  {
WWB_UNROLL(1)
    for (int j = lane; j < l.n; j += Grp::kLanes) {
      one_copy();
      sin4_tail(x, l.at(j));
    }
    syncwarp();
    if (p.sintailpar[0] < 0.5f) {
      // TAU1's terms: they do not feed the next step of the tail, so they are formed side by side.
      const float dely = x.w[L.tail + 7 * kJtot];
WWB_UNROLL(1)
      for (int e = lane; e < l.n * kJtot; e += Grp::kLanes) {
        const int n = e / kJtot, k = l.at(n), j = e - n * kJtot;
        float* const t = x.s(k, L.jt);
        const float w = (j == 0 || j == kJtot - 1) ? 0.5f : 1.0f;
        const float lev = p.sintailpar[2] > 0.0f ? t[kLev + j] : x.sh[k].levtail0;
        t[kZb + j] = w * t[kZb + j] * t[kUs + j] * lev * dely * x.w[L.tail + kJtot + j] /
                       x.w[L.tail + j];
      }
      syncwarp();
    }
WWB_UNROLL(1)
    for (int j = lane; j < l.n; j += Grp::kLanes) {
      one_copy();
      const int k = l.at(j);
      SrceSh& s = x.sh[k];
      float tauhf = s.tauhf;
      if (p.sintailpar[0] < 0.5f) tauhf = sum4(x.s(k, L.jt) + kZb, kJtot, 0.0f);
      float cp, sp;
      sincosf_i(s.usdirpl, &sp, &cp);
      float twx = s.stress[0] + tauhf * cp;
      float twy = s.stress[1] + tauhf * sp;
      const float tauw = sqrt_f(twx * twx + twy * twy);
      const float ust2b = max_r(s.r.ustar, kEps2);
      const float ust2 = ust2b * ust2b;
      const float tauwb = min_r(tauw, max_r(ust2 - kEps1, kEps2Sq));
      if (tauwb < tauw) {
        twx = twx * tauwb / tauw;
        twy = twy * tauwb / tauw;
      }
      s.tauwx = twx;
      s.tauwy = twy;
    }
  }
}

WWB_PD bool finite_f(float v) { return fabs_f(v) <= 3.402823466e38f; }

/// W3SIN4 (w3src4md.F90:423-1003) of the listed slots with W3SRCE's arguments (:1100, :1239, :2007):
/// VDIN, LLWS, TAUWX/Y, TAUWAX/Y. VSIN = VDIN * SPEC is formed where it is read (the spectrum does not
/// change before that).
template <class G>
WWB_PD void srce_sin4(const Grp& c, const G& x, const SlotList& l) {
  const SrceLayout& L = *x.L;
  const st4::Params& p = *x.q;
  const Fields& f = *x.f;
  const int nk = L.nk, nth = x.nth();
  const Sin4At at = sin4_at(L);
  // 1. Preparations (:600-675).
  each_row(c, l, nk, [&](int k, int ik) {
    const SrceSh& s = x.sh[k];
    const float e = row_sum(x.s(k, L.spec), ik, nth);
    const float kis = x.s(k, L.wn1)[ik], cg = x.s(k, L.cg1)[ik];
    const float sig2is = f.sig2[ik * nth], sigk = f.sig[ik + 1];
    const float const0 = (p.bbeta / kKappa2) * s.drat;
    float* const t = x.tr(k) + ik;
    t[at.cm] = kis / sig2is;
    t[at.const2] = f.dden2[ik * nth] / cg * kGrav / (sigk / kis * s.drat);
    t[at.cnst] = sig2is * const0;
    t[at.zcn] = dm::logf_q(kis * s.r.z0);
    t[at.swv] = -(p.sswellf[4] * s.drat * 2.0f * kis * sqrt_f(kTwoNuAir * sig2is));
    t[at.swt] = -(s.drat * p.sswellf[0] * 16.0f * (sig2is * sig2is) / kGrav);
    t[at.tu] = e * (sigk * sigk) * f.dden[ik] / cg;
    t[at.ta] = e * f.dden[ik] / cg;
  });
  if (p.sintailpar[0] < 0.5f)
    each_row(c, l, kJtot, [&](int k, int j) {
      x.s(k, L.jt)[kGz + j] = kGrav * x.sh[k].r.z0 / x.w[L.tail + 4 * kJtot + j];
    });
  c.sync();
  each_chain(c, 0, l, [&](int k) {
    SrceSh& s = x.sh[k];
    const float* const t = x.tr(k);
    const float ustar = s.r.ustar;
    const float const1 = p.bbeta / kKappa2;
    const float z0visc = kZ0viscNum / max_r(ustar, 0.0001f);
    const float z0noz = max_r(z0visc, p.zz0rat * s.r.z0);
    float uorb = 0.0f, aorb = 0.0f;
WWB_UNROLL(4)
    for (int ik = 0; ik < nk; ++ik) {
      uorb = uorb + t[at.tu + ik];
      aorb = aorb + t[at.ta + ik];
    }
    uorb = 2.0f * sqrt_f(uorb);
    const float aorb1 = 2.0f * dm::powf(aorb, 1.0f - 0.5f * p.sswellf[5]);
    const float re = 4.0f * uorb * aorb1 / kNuAir;
    float pturb, pvisc;
    if (p.sswellf[3] > 0.0f) {
      if (p.sswellf[6] > 0.0f) {
        const float smooth = 0.5f * dm::tanhf((re - p.sswellf[3]) / p.sswellf[6]);
        pturb = (0.5f + smooth);
        pvisc = (0.5f - smooth);
      } else if (re <= p.sswellf[3]) {
        pturb = 0.0f;
        pvisc = 1.0f;
      } else {
        pturb = 1.0f;
        pvisc = 0.0f;
      }
    } else {
      pturb = 1.0f;
      pvisc = 1.0f;
    }
    float fw, fu, fud;
    if (p.sswellf[1] == 0.0f) {
      fw = fabs_f(p.sswellf[2]);
      fu = 0.0f;
      fud = 0.0f;
    } else {
      fu = fabs_f(p.sswellf[2]);
      fud = p.sswellf[1];
      aorb = 2.0f * sqrt_f(aorb);
      const float xi = (dm::log10f(max_r(aorb / z0noz, 3.0f)) - kAbMin) / p.delab;
      const int ind = min_i(st4::kSizeFwTable - 1, fint(xi));
      const float deli1 = min_r(1.0f, xi - static_cast<float>(ind));
      const float deli2 = 1.0f - deli1;
      fw = f.fwtable[ind] * deli2 + f.fwtable[ind + 1] * deli1;
    }
    float ustarsigma = 0.0f;
    if (p.stab3) {
      float usigma;
      if (isnan_f(s.in.as)) {
        usigma = 0.0f;
      } else {
        usigma = max_r(0.0f, -0.025f * s.in.as);
      }
      ustarsigma = (1.0f + s.in.u10abs / (10.0f + s.in.u10abs)) * usigma;
    }
    s.const1 = const1;
    s.fwuorb = fw * uorb;
    s.pturb = pturb;
    s.pvisc = pvisc;
    s.fu = fu;
    s.fud = fud;
    s.ustarsigma = ustarsigma;
    for (int i = 0; i < 3; ++i)
      for (int j = 0; j < 2; ++j) s.ss[i][j] = s.sn[i][j] = 0.0f;
  });
  // With TTAUWSHELTER = 0 the running stress enters as TAU - 0 * STRESS, which is TAU itself as
  // long as TAU is not a zero (whose sign it could change) and STRESS is finite (checked after the
  // sums): the friction velocity, its direction and so every frequency are then independent.
  each_chain(c, 1, l, [&](int k) {
    SrceSh& s = x.sh[k];
    const float ust = s.r.ustar;
    const float taux = (ust * ust) * s.cosw, tauy = (ust * ust) * s.sinw;
    const bool par = !p.stab3 && p.ttauwshelter == 0.0f && taux != 0.0f && tauy != 0.0f;
    s.scan_par = par ? 1 : 0;
    if (par) {
      s.ust = ust;
      s.taux = taux;
      s.tauy = tauy;
      s.ustp = min_r(dm::powf((taux * taux + tauy * tauy), 0.25f), max_r(ust, 0.3f));
      float sn, cs;
      sincosf_i(dm::atan2f(tauy, taux), &sn, &cs);
      s.cosu = cs;
      s.sinu = sn;
    }
  });
  c.sync();
  // 2. The stress scan over IK (:696-797).
  SlotList par{}, ser{};
WWB_UNROLL(1)
  for (int j = 0; j < l.n; ++j) {
    if (x.sh[l.at(j)].scan_par) par.add(l.at(j));
    else ser.add(l.at(j));
  }
  if (par.n) {
    const int R = (L.nspec + 3) & ~3;
    const bool plain = scan_plain(p);
    struct Slot {
      const float* spec;
      float *vdin, *t;
      const float* tk;
      unsigned char *llws, *neg;
      float ustar, ustp, cosu, sinu;
      Swell sw;
    };
    bins(c, par, L.nspec, [&](int k) {
      const SrceSh& s = x.sh[k];
      return Slot{x.s(k, L.spec), x.gs(k, L.vdin), x.tr(k), x.tr(k), x.llws(k),
                  reinterpret_cast<unsigned char*>(x.tr(k) + 2 * R), s.r.ustar, s.ustp, s.cosu, s.sinu,
                  Swell{s.fwuorb, s.fu, s.fud, s.pturb, s.pvisc}};
    }, [&](const Slot& s, int i) {
      const int ik = x.row(i);
      const ScanK q = scan_k(x, at, s.tk, ik, s.ustp);
      const int ith = i - ik * nth;
      const float ecos = x.ecos(ik)[ith], esin = x.esin(ik)[ith];
      const float coswind = (ecos * s.cosu + esin * s.sinu);
      int lw;
      bool ok = plain;
      float dst = scan_bin_q(p, s.sw, q, s.ustar, s.ustp, coswind, &lw, &ok);
      if (!ok) dst = scan_bin(p, s.sw, q, s.ustar, s.ustp, coswind, &lw);
      s.vdin[i] = dst;
      s.llws[i] = static_cast<unsigned char>(lw);
      const float temp2 = q.const2 * dst * s.spec[i];
      s.t[i] = temp2 * ecos;
      s.t[R + i] = temp2 * esin;
      s.neg[i] = dst < 0.0f ? 1 : 0;
    });
    c.sync();
    each_chain_of(c, 0, 4, par, [&](int r, int k) {
        const float* const t = x.tr(k);
        const float v = sum_flagged(t + (r & 1) * R, reinterpret_cast<const unsigned char*>(t + 2 * R),
                                    L.nspec, static_cast<unsigned>(r >> 1), 0.0f);
        x.sh[k].sums[r] = v;
        (r < 2 ? x.sh[k].ss : x.sh[k].sn)[2][r & 1] = v;
    });
    c.sync();
WWB_UNROLL(1)
    for (int j = 0; j < par.n; ++j) {
      const SrceSh& s = x.sh[par.at(j)];
      if (!finite_f(s.sums[0]) || !finite_f(s.sums[1])) ser.add(par.at(j));
    }
  }
  if (ser.n) {
    c.sync();
    scan_serial(c, x, ser, at);
    c.sync();
  }
  // 3. TAUWX and TAUWY enter the next step's fluxes and W3SPR4 only: the tail warp forms them beside the
  // next step's DIA and W3SDS4.
  if (x.box != nullptr) {
    if (c.tid == 0) x.box->l = l;
    c.tail_go();
  } else {
    sin4_close(0, x, l, [] {});
  }
}

// ------------------------------------------------------------------------- the DIA (W3SNL1)
/// The step's DIA (:1259-1263) with KDMEAN = WNMEAN * DEPTH for the listed slots (the arithmetic of
/// snl1_rowshift_kernel): VSNL and VDNL. UE, SA1, SA2 of as many slots as fit sit in the transient
/// region; DA1P, DA1M, DA2P, DA2M and DA1C + DA2C in the slot's global scratch (DA1C and DA2C are read
/// back only at their own bin, so their sum is kept, the same two roundings).
template <class G>
WWB_PD void srce_dia(const Grp& c, const G& x, const SlotList& all) {
  const SrceLayout& L = *x.L;
  const Snl1Dev& p = *x.n;
  const int nth = x.nth(), nfr = p.nfr, nfrhgh = p.nfrhgh, nfrchg = p.nfrchg;
  const int nspec = L.nspec, nk = L.nk;
  const int A4 = (L.alen + 3) & ~3, U4 = ((nfrhgh + 1) * nth + 3) & ~3;
  const int per = srce_trans_floats(L, x.ns) / L.dia;
  const float dal1 = p.dal1, dal2 = p.dal2, dal3 = p.dal3;
WWB_UNROLL(1)
  for (int j0 = 0; j0 < all.n; j0 += per) {
    SlotList l{};
WWB_UNROLL(1)
    for (int j = j0; j < all.n && j < j0 + per; ++j) l.add(all.at(j));
    // Position j of a slot in this round picks its part of the region.
    auto ue_of = [&](int k) {
      int j = 0;
      for (int m = 1; m < kSlots; ++m) j = (m < l.n && l.at(m) == k) ? m : j;
      return x.t + j * L.dia;
    };
    each_row(c, l, nth, [&](int k, int i) {
      float* const ue = ue_of(k);
      ue[i] = 0.0f;
      ue[U4 + i] = ue[U4 + A4 + i] = 0.0f;
      float* const da = x.gs(k, L.da);
      for (int m = 0; m < 4; ++m) da[m * A4 + i] = 0.0f;
    });
    each_row(c, l, nk, [&](int k, int ik) {
      ue_of(k)[U4 + 2 * A4 + ik] = kTpiInv / p.sig[ik] * x.s(k, L.cg1)[ik];
    });
    c.sync();
    struct SlotA {
      float* ue;
      const float *spec, *conx;
    };
    bins(c, l, nspec, [&](int k) {
      float* const ue = ue_of(k);
      return SlotA{ue + nth, x.s(k, L.spec), ue + U4 + 2 * A4};
    }, [&](const SlotA& s, int i) { s.ue[i] = s.spec[i] / s.conx[x.row(i)]; });
    c.sync();
    each_row(c, l, nth, [&](int k, int col) {
      float* const ue = ue_of(k);
      float t = ue[nfr * nth + col];
WWB_UNROLL(1)
      for (int r = nfr + 1; r <= nfrhgh; ++r) {
        t = t * p.fachfe;
        ue[r * nth + col] = t;
      }
    });
    // Section 1: CONS (snl1_team.hpp:383-390).
    each_chain(c, 7, l, [&](int k) {
      SrceSh& s = x.sh[k];
      const float kdmean = s.r.wnmean * s.depth;
      const float x0 = p.kdcon * kdmean;
      const float xx = (x0 < p.kdmn) ? p.kdmn : x0;
      const float y0 = p.snls3 * xx;
      const float x2 = (-1.e15f < y0) ? y0 : -1.e15f;
      s.cons = p.snlc1 * (1.0f + p.snls1 / xx * (1.0f - p.snls2 * xx) * dm::expf(x2));
    });
    c.sync();
    // The eight wrapped directions of a bin: constant for a thread.
    struct Cols {
      int ith, cc[8];
    };
    auto cols = [&](int ith) {
      Cols q;
      q.ith = ith;
      for (int n = 0; n < 8; ++n) {
        const int v = ith + p.shift[n];
        q.cc[n] = v < 0 ? v + nth : (v >= nth ? v - nth : v);
      }
      return q;
    };
    dirs(c, l, nth, nfrchg, cols, [&](const Cols& q, int k, int ifr0) {
      float* const ue = ue_of(k);
      const int* const cc = q.cc;
      const float* const u1 = ue + p.ifrow[0 * nfrchg + ifr0] * nth;
      const float* const u2 = ue + p.ifrow[1 * nfrchg + ifr0] * nth;
      const float* const u3 = ue + p.ifrow[2 * nfrchg + ifr0] * nth;
      const float* const u4 = ue + p.ifrow[3 * nfrchg + ifr0] * nth;
      const int isp = ifr0 * nth + q.ith, o = isp + nth;
      const float e00 = ue[o];
      const float ep1 = p.awg[0] * u2[cc[1]] + p.awg[1] * u2[cc[0]] +
                        p.awg[2] * u1[cc[1]] + p.awg[3] * u1[cc[0]];
      const float em1 = p.awg[4] * u4[cc[7]] + p.awg[5] * u4[cc[6]] +
                        p.awg[6] * u3[cc[7]] + p.awg[7] * u3[cc[6]];
      const float ep2 = p.awg[0] * u2[cc[5]] + p.awg[1] * u2[cc[4]] +
                        p.awg[2] * u1[cc[5]] + p.awg[3] * u1[cc[4]];
      const float em2 = p.awg[4] * u4[cc[3]] + p.awg[5] * u4[cc[2]] +
                        p.awg[6] * u3[cc[3]] + p.awg[7] * u3[cc[2]];
      const float ca = x.sh[k].cons * p.af11_row[ifr0];
      const float factor = ca * e00;
      const float sa1a = e00 * (ep1 * dal1 + em1 * dal2);
      const float sa1b = sa1a - ep1 * em1 * dal3;
      const float sa2a = e00 * (ep2 * dal1 + em2 * dal2);
      const float sa2b = sa2a - ep2 * em2 * dal3;
      ue[U4 + o] = factor * sa1b;
      ue[U4 + A4 + o] = factor * sa2b;
      float* const da = x.gs(k, L.da) + o;
      if (isp < nspec) da[4 * A4 - nth] = ca * (sa1a + sa1b) + ca * (sa2a + sa2b);
      da[0] = factor * (dal1 * e00 - dal3 * em1);
      da[A4] = factor * (dal2 * e00 - dal3 * ep1);
      da[2 * A4] = factor * (dal1 * e00 - dal3 * em2);
      da[3 * A4] = factor * (dal2 * e00 - dal3 * ep2);
    });
    c.sync();
    dirs(c, l, nth, nk, cols, [&](const Cols& q, int k, int ifr0) {
      const float* const ue = ue_of(k);
      const float* const sa = ue + U4;
      const float* const da = x.gs(k, L.da);
      const int* const cc = q.cc;
      const int o5 = p.ifrow[4 * nfrchg + ifr0] * nth;
      const int o6 = p.ifrow[5 * nfrchg + ifr0] * nth;
      const int o7 = p.ifrow[6 * nfrchg + ifr0] * nth;
      const int o8 = p.ifrow[7 * nfrchg + ifr0] * nth;
      const int isp = ifr0 * nth + q.ith, o = isp + nth;
      // DA*P rows 5, 6 and DA*M rows 7, 8 of the two interactions, all on their way at once.
      const float *const d5 = da + o5, *const d6 = da + o6, *const d7 = da + A4 + o7,
                  *const d8 = da + A4 + o8;
      const float p65 = d6[cc[5]], p64 = d6[cc[4]], p55 = d5[cc[5]], p54 = d5[cc[4]];
      const float q61 = d6[2 * A4 + cc[1]], q60 = d6[2 * A4 + cc[0]], q51 = d5[2 * A4 + cc[1]],
                  q50 = d5[2 * A4 + cc[0]];
      const float m83 = d8[cc[3]], m82 = d8[cc[2]], m73 = d7[cc[3]], m72 = d7[cc[2]];
      const float n87 = d8[2 * A4 + cc[7]], n86 = d8[2 * A4 + cc[6]], n77 = d7[2 * A4 + cc[7]],
                  n76 = d7[2 * A4 + cc[6]];
      const float dc = da[4 * A4 + isp];
      const float *const s5 = sa + o5, *const s6 = sa + o6, *const s7 = sa + o7, *const s8 = sa + o8;
      x.gs(k, L.vsnl)[isp] = ue[U4 + 2 * A4 + ifr0] * (-2.0f * (sa[o] + sa[A4 + o]) +
                             p.awg[0] * (s6[cc[5]] + s6[A4 + cc[1]]) +
                             p.awg[1] * (s6[cc[4]] + s6[A4 + cc[0]]) +
                             p.awg[2] * (s5[cc[5]] + s5[A4 + cc[1]]) +
                             p.awg[3] * (s5[cc[4]] + s5[A4 + cc[0]]) +
                             p.awg[4] * (s8[cc[3]] + s8[A4 + cc[7]]) +
                             p.awg[5] * (s8[cc[2]] + s8[A4 + cc[6]]) +
                             p.awg[6] * (s7[cc[3]] + s7[A4 + cc[7]]) +
                             p.awg[7] * (s7[cc[2]] + s7[A4 + cc[6]]));
      x.gs(k, L.vdnl)[isp] = -2.0f * dc + p.swg[0] * (p65 + q61) + p.swg[1] * (p64 + q60) +
                             p.swg[2] * (p55 + q51) + p.swg[3] * (p54 + q50) +
                             p.swg[4] * (m83 + n87) + p.swg[5] * (m82 + n86) +
                             p.swg[6] * (m73 + n77) + p.swg[7] * (m72 + n76);
    });
    c.sync();
  }
}

// ------------------------------------------------------------------------------------ W3SDS4
WWB_PD int first_bit(unsigned m) {
#if defined(__CUDA_ARCH__)
  return __ffs(static_cast<int>(m)) - 1;
#else
  return __builtin_ctz(m);
#endif
}

/// BTH of the saturation (:2262-2290) for up to NS listed slots. A thread takes a bin of every slot, so
/// the weights and indices are read once for all of them; a missing slot repeats the first one.
template <int NS, class G>
WWB_PD void sat_sums(const Grp& c, const G& x, const SlotList& l, int rows, int ik1) {
  const SrceLayout& L = *x.L;
  const Fields& f = *x.f;
  const int nth = x.nth(), nspec = L.nspec, ld = f.sat_ld;
  const float dth = x.q->dth;
  const float* spec[NS];
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
  for (int m = 0; m < NS; ++m) spec[m] = x.s(l.at(m < l.n ? m : 0), L.spec);
WWB_UNROLL(1)
  for (int i = c.tid; i < nspec; i += c.nthr) {
    one_copy();
    const int ik0 = x.row(i), ith0 = i - ik0 * nth;
    const int row = ik0 * nth - 1;
    const float* sw = f.satw_t + ith0;
    const int* si = f.sati_t + ith0;
    float v[NS] = {};
    if (ik0 + 1 >= ik1) {
WWB_UNROLL(6)
      for (int j = 0; j < rows; ++j) {
        const float w = *sw;
        const int o = row + *si;
        sw += ld;
        si += ld;
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
        for (int m = 0; m < NS; ++m) v[m] = v[m] + w * spec[m][o];
      }
    }
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
    for (int m = 0; m < NS; ++m) {
      if (m >= l.n) break;
      const int k = l.at(m);
      const float kx = x.s(k, L.wn1)[ik0];
      const float facsat = (f.sig[ik0 + 1] * ((kx * kx) * kx)) * dth;
      x.tr(k)[i] = ik0 + 1 >= ik1 ? v[m] * facsat : 0.0f;
    }
  }
}

/// Wave-turbulence interaction and the cumulative effect (:2533-2575) for up to NS listed slots; mask_at
/// and ren_at: the slots' block masks and (SSDSC(3) > 0) renewal sums in the transient region. A thread
/// takes a bin of every slot: CUMULW's row is read once for all of them and BRLAMBDA is a broadcast. The
/// sums grow with the frequency: the warps take the bins from the top, forwards and backwards in turn.
template <int NS, class G>
WWB_PD void sds4_turb(const Grp& c, const G& x, const SlotList& l, bool blocks, int dikcumul, int ik1,
                      int mask_at, int ren_at) {
  constexpr int NTH = G::kNth;
  const SrceLayout& L = *x.L;
  const Fields& f = *x.f;
  const float* ssdsc = x.q->ssdsc;
  const int nk = L.nk, nth = x.nth(), nspec = L.nspec;
  const float sc2 = ssdsc[2], dvc = ssdsc[20] * 4.0f;
  const float* brl[NS];
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
  for (int j = 0; j < NS; ++j) brl[j] = x.tr(l.at(j < l.n ? j : 0));
  const int nch = (nspec + Grp::kLanes - 1) / Grp::kLanes, nw = c.nwarp();
WWB_UNROLL(1)
  for (int round = 0; round * nw < nch; ++round) {
    const int e = nch - 1 - (round * nw + (round & 1 ? nw - 1 - c.warp() : c.warp()));
    const int i = e * Grp::kLanes + c.lane();
    if (e < 0 || i >= nspec) continue;
    one_copy();
    const int ik0 = x.row(i), ik = ik0 + 1, ith0 = i - ik0 * nth;
    if (ik < ik1) continue;
    float ren[NS] = {};
    if (sc2 < 0.0f) {
WWB_UNROLL(1)
      for (int ik2 = ik1; ik2 <= ik - dikcumul; ++ik2) {
        one_copy();
        unsigned m[NS], any = 0;
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
        for (int j = 0; j < NS; ++j) {
          m[j] = j < l.n ? reinterpret_cast<const unsigned*>(brl[j] + mask_at)[ik2 - 1] : 0u;
          any |= m[j];
        }
        if (any == 0) continue;
        const int is2 = (ik2 - 1) * nth;
        float v[NS] = {};
        // CUMULW(IS2+J, IS) as a function of IK2, IK and J - ITH where the table is one (f.cumt), else
        // the transposed table: consecutive IS are consecutive in both.
        if (NTH != 0 && NTH % 12 == 0 && blocks && f.cumt != nullptr) {
          const float* const cw = f.cumt + ((ik2 - 1) * nk + ik0) * (2 * NTH - 1) + (NTH - 1 - ith0);
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
          for (int b0 = 0; b0 < NTH / 4; b0 += 3) {
            if ((any >> b0 & 7u) == 0) continue;
            float q[12];
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
            for (int d = 0; d < 12; ++d) q[d] = cw[4 * b0 + d];
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
            for (int b = 0; b < 3; ++b) {
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
              for (int j = 0; j < NS; ++j) {
                if (m[j] & (1u << (b0 + b))) {
                  const F4 r = ld4(brl[j] + is2 + 4 * (b0 + b));
                  v[j] = v[j] + q[4 * b] * r.a;
                  v[j] = v[j] + q[4 * b + 1] * r.b;
                  v[j] = v[j] + q[4 * b + 2] * r.c;
                  v[j] = v[j] + q[4 * b + 3] * r.d;
                }
              }
            }
          }
        } else {
          const bool toe = f.cumt != nullptr;
          const float* const cw =
              toe ? f.cumt + (static_cast<size_t>(ik2 - 1) * nk + ik0) * (2 * nth - 1) + (nth - 1 - ith0)
                  : f.cumulw + static_cast<size_t>(is2) * f.cumulw_ld + i;
          const size_t step = toe ? 1 : f.cumulw_ld;
          const int width = blocks ? 4 : nth;
WWB_UNROLL(1)
          for (; any; any &= any - 1u) {
            const int b = first_bit(any);
WWB_UNROLL(1)
            for (int d = width * b; d < width * b + width; ++d) {
              const float q = cw[static_cast<size_t>(d) * step];
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
              for (int j = 0; j < NS; ++j)
                if (m[j] >> b & 1) v[j] = v[j] + q * brl[j][is2 + d];
            }
          }
        }
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
        for (int j = 0; j < NS; ++j)
          if (m[j]) ren[j] = ren[j] + v[j];
      }
    }
    const float sig2 = f.sig[ik] * 2.0f, ecos = f.ecos[ith0], esin = f.esin[ith0];
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
    for (int j = 0; j < NS; ++j) {
      if (j >= l.n) break;
      const int k = l.at(j);
      const SrceSh& s = x.sh[k];
      const float kx = x.s(k, L.wn1)[ik0];
      const float facturb2 = -((sig2 * kx) * s.facturb);
      const float dvisc = -((dvc * kx) * kx);
      const float renewalfreq = sc2 > 0.0f ? brl[j][ren_at + ik0] : ren[j];
      const float coswind = ecos * s.cosus + esin * s.sinus;
      const float dturb = facturb2 * max_r(coswind, 0.0f);
      const float diag2 = (sc2 * renewalfreq + dturb) + dvisc;
      float* const vdds = x.gs(k, L.vdds) + i;
      float* const vsds = x.gs(k, L.vsds) + i;
      *vdds = *vdds + diag2;
      *vsds = *vsds + x.s(k, L.spec)[i] * diag2;
    }
  }
}

/// W3SDS4 (w3src4md.F90:2043-2659) of the listed slots: VSDS, VDDS, WHITECAP. BRLAMBDA stays in the
/// slot's transient region (BTH before it, in place), the NK arrays behind it. The libmvec loops
/// (:2315, :2500, :2509) use scalar powf/expf in every lane.
template <class G>
WWB_PD void srce_sds4(const Grp& c, const G& x, const SlotList& l) {
  const SrceLayout& L = *x.L;
  const st4::Params& p = *x.q;
  const Fields& f = *x.f;
  const int nk = L.nk, nth = x.nth(), nspec = L.nspec;
  const int R = (nspec + 3) & ~3, K = (nk + 3) & ~3;
  const float* ssdsc = p.ssdsc;
  const float zero = 0.0f, one = 1.0f;
  enum { kBth0 = 0, kA1, kA2, kA3, kCoef4, kCoef5, kBrm12, kRen, kMss1, kMss2, kMss3, kMss4, kB1, kB2, kB3, kB4, kB5, kB6 };
  static_assert(kB6 < kNkWork, "kNkWork NK arrays");
  auto brl_of = [&](int k) { return x.tr(k); };
  auto nka = [&](int k, int j) { return x.tr(k) + R + j * K; };
  const int dikcumul = nint(p.ssdsbrf1 / (p.xfr - one));
  const int ik1 = p.ig1 ? nint(p.igpars5) + 1 : 1;
  const float dth = p.dth;
  each_chain(c, 0, l, [&](int k) {
    SrceSh& s = x.sh[k];
    s.facturb = (((ssdsc[4] * (s.r.ustar * s.r.ustar)) / kGrav) * s.in.dair) / kDwat;
    float sn, cs;
    dm::sincosf(s.r.usdir, &sn, &cs);
    s.sinus = sn;
    s.cosus = cs;
  });
  const int sdscase = nint(ssdsc[0]);
  if (sdscase == 1) {
    // 2.a.1 Saturation (:2262-2290).
    if (p.ssdsdth < 180.0f) {
      // Rows of SATWEIGHTS past nsat_eff are all zero for one and the same bin: adding 0 * A once has
      // the effect of adding it for each of them.
      const int rows = f.nsat_eff < f.nsat ? f.nsat_eff + 1 : f.nsat;
WWB_UNROLL(1)
      for (int j = 0; j < l.n; j += kTogether) {
        one_copy();
        const SlotList g = l.part(j, kTogether);
        if (g.n == 1) sat_sums<1>(c, x, g, rows, ik1);
        else sat_sums<kTogether>(c, x, g, rows, ik1);
      }
      c.sync();
    }
    each_row(c, l, nk, [&](int k, int ik0) {
      const int ik = ik0 + 1, is0 = ik0 * nth;
      float b0 = zero;
      const float kx = x.s(k, L.wn1)[ik0];
      if (ik >= ik1) {
        if (p.ssdsdth >= 180.0f) {
          const float facsat = (f.sig[ik] * ((kx * kx) * kx)) * dth;
          b0 = row_sum(x.s(k, L.spec), ik0, nth) * facsat;
        } else {
          // MAXVAL as gfortran lowers it: the first element >= -Inf, then strictly greater.
          const float* const bth = brl_of(k);
          float lim = -dm::asfloat(0x7f800000u);
          int i = is0;
          bool found = false;
WWB_UNROLL(1)
          for (; i < is0 + nth; ++i) {
            if (bth[i] >= lim) {
              lim = bth[i];
              ++i;
              found = true;
              break;
            }
          }
          if (!found) lim = dm::asfloat(0x7fc00000u);
WWB_UNROLL(1)
          for (; i < is0 + nth; ++i)
            if (bth[i] > lim) lim = bth[i];
          b0 = lim;
        }
        // 2.a.2 Spontaneous breaking (:2291-2331), the factors of one IK.
        float miche;
        if (p.ssdsbm[0] == one) {
          miche = one;
        } else {
          const float xx = dm::tanhf(min_r(kx * x.sh[k].depth, 10.0f));
          const float t =
              xx * (p.ssdsbm[1] + xx * (p.ssdsbm[2] + xx * (p.ssdsbm[3] + xx * p.ssdsbm[4])));
          miche = t * t;
        }
        const float coef1 = p.ssdsbr * miche;
        const float m = max_r(b0 / coef1 - one, zero);
        nka(k, kA1)[ik0] = coef1;
        nka(k, kA2)[ik0] = ((ssdsc[1] * f.sig[ik]) * ssdsc[5]) * (m * m);
        nka(k, kA3)[ik0] = ((ssdsc[1] * f.sig[ik]) * (one - ssdsc[5])) / (coef1 * coef1);
      }
      nka(k, kBth0)[ik0] = b0;
      nka(k, kBrm12)[ik0] = zero;
    });
    c.sync();
    const float epsr = sqrt_f(p.ssdsbr);
    struct Slot {
      float* brl;
      const float *bth0, *a1, *a2, *a3, *spec;
      float *vdds, *vsds;
    };
    const bool iso = p.ssdsdth >= 180.0f;
    bins(c, l, nspec, [&](int k) {
      return Slot{brl_of(k), nka(k, kBth0), nka(k, kA1), nka(k, kA2), nka(k, kA3), x.s(k, L.spec),
                  x.gs(k, L.vdds), x.gs(k, L.vsds)};
    }, [&](const Slot& s, int i) {
      const int ik0 = x.row(i);
      float bth = zero, dd = zero;
      if (ik0 + 1 >= ik1) {
        bth = iso ? s.bth0[ik0] : s.brl[i];
        // Below the threshold the power of 0 is 0 (SSDSP > 0): most warps have no bin above it.
        const float over = max_r(bth - s.a1[ik0], zero);
        dd = s.a2[ik0] + s.a3[ik0] * (over == zero && p.ssdsp > zero ? zero : powf_i(over, p.ssdsp));
      }
      const float m = max_r(sqrt_f(bth) - epsr, zero);
      float pbi = m * m;
      pbi = pbi * 28.16f;
      s.brl[i] = pbi / kTwoPiSq;
      s.vdds[i] = dd;
      s.vsds[i] = dd * s.spec[i];
    });
    c.sync();
  } else if (sdscase == 2) {
    // 2.b Filipot et al. (:2338-2477). E1 = kB1, DK = kB2, the serial part's arrays behind.
    each_row(c, l, nk, [&](int k, int ik0) {
      const int ik = ik0 + 1;
      float e = zero, dk = zero;
      if (ik >= ik1) {
        const float* const a = x.s(k, L.spec) + ik0 * nth;
WWB_UNROLL(1)
        for (int ith = 0; ith < nth; ++ith) e = e + (a[ith] * f.sig[ik]) * dth;
        dk = f.dden[ik0] / ((dth * f.sig[ik]) * x.s(k, L.cg1)[ik0]);
      }
      nka(k, kB1)[ik0] = e;
      nka(k, kB2)[ik0] = dk;
      nka(k, kBrm12)[ik0] = zero;
    });
    c.sync();
    each_chain(c, 0, l, [&](int k) {
      const float depth = x.sh[k].depth;
      const float* const kk = x.s(k, L.wn1);
      float* const e1 = nka(k, kB1);
      float* const dk = nka(k, kB2);
      float* const hs = nka(k, kB3);
      float* const kbar = nka(k, kB4);
      float* const efdf = nka(k, kB5);
      float* const dck = nka(k, kB6);
      float* const qb = nka(k, kA1);
      float* const s1 = nka(k, kA2);
      float* const s2 = nka(k, kA3);
      int* const ntimes = reinterpret_cast<int*>(nka(k, kMss1));
      int* const iksup = reinterpret_cast<int*>(nka(k, kMss2));
      int id = nint(depth);
      if (id > st4::kNdtab) id = st4::kNdtab;
      if (id < 1) id = 1;
      int nkl = 0;
WWB_UNROLL(1)
      for (int i = 0; i < nk; ++i) hs[i] = efdf[i] = kbar[i] = zero;
WWB_UNROLL(1)
      for (int ikl = 1; ikl <= nk; ++ikl) {
        iksup[ikl - 1] = f.iktab[(ikl - 1) + (id - 1) * f.iktab_ld];
        if (iksup[ikl - 1] <= nk) {
          float v = zero;
WWB_UNROLL(1)
          for (int i = ikl; i <= iksup[ikl - 1] - 1; ++i) v = v + e1[i - 1] * dk[i - 1];
          efdf[ikl - 1] = v;
          if (efdf[ikl - 1] != zero) {
            float w = zero;
WWB_UNROLL(1)
            for (int i = ikl; i <= iksup[ikl - 1] - 1; ++i) w = w + (kk[i - 1] * e1[i - 1]) * dk[i - 1];
            kbar[ikl - 1] = w / efdf[ikl - 1];
          } else {
            kbar[ikl - 1] = zero;
          }
          hs[ikl - 1] = 4.0f * sqrt_f(efdf[ikl - 1]);
          nkl = nkl + 1;
        }
      }
WWB_UNROLL(1)
      for (int i = 0; i < nk; ++i) dck[i] = qb[i] = zero;
WWB_UNROLL(1)
      for (int ikl = 1; ikl <= nkl; ++ikl) {
        const float kb = kbar[ikl - 1];
        if (hs[ikl - 1] != zero && kb != zero) {
          int ikd = fint(roundf(dm::logf(kb * depth) / kLogFacKd1) + static_cast<float>(kFacKd2));
          int ikhs = fint(one + roundf((kb * hs[ikl - 1]) / kDkhs));
          if (ikd > st4::kNkd) ikd = st4::kNkd;
          else if (ikd < 1) ikd = 1;
          if (ikhs > st4::kNkhs) ikhs = st4::kNkhs;
          else if (ikhs < 1) ikhs = 1;
          dck[ikl - 1] = (dm::powf(kb, -2.5f) * (kb / kTwoPi)) *
                         f.dcki[(ikhs - 1) + (ikd - 1) * st4::kNkhs];
          qb[ikl - 1] = f.qbi[(ikhs - 1) + (ikd - 1) * st4::kNkhs];
        } else {
          dck[ikl - 1] = zero;
          qb[ikl - 1] = zero;
        }
      }
WWB_UNROLL(1)
      for (int i = 0; i < nk; ++i) {
        s1[i] = s2[i] = zero;
        ntimes[i] = 0;
      }
WWB_UNROLL(1)
      for (int ikl = 1; ikl <= nkl; ++ikl) {
        if (efdf[ikl - 1] > zero) {
WWB_UNROLL(1)
          for (int i = ikl; i <= iksup[ikl - 1]; ++i)
            s1[i - 1] = s1[i - 1] + (dck[ikl - 1] * e1[i - 1]) / efdf[ikl - 1];
WWB_UNROLL(1)
          for (int i = ikl; i <= iksup[ikl - 1]; ++i)
            s2[i - 1] = s2[i - 1] + (qb[ikl - 1] * e1[i - 1]) / efdf[ikl - 1];
WWB_UNROLL(1)
          for (int i = ikl; i <= iksup[ikl - 1]; ++i) ntimes[i - 1] = ntimes[i - 1] + 1;
        }
      }
WWB_UNROLL(1)
      for (int i = 0; i < nk; ++i) {
        if (ntimes[i] > 0) {
          s1[i] = s1[i] / static_cast<float>(ntimes[i]);
          s2[i] = s2[i] / static_cast<float>(ntimes[i]);
        } else {
          s1[i] = s2[i] = zero;
        }
      }
WWB_UNROLL(1)
      for (int ik = 1; ik <= nk; ++ik) s1[ik - 1] = s1[ik - 1] / f.sig[ik];
    });
    c.sync();
    // DDIAG and PB2 are one value per IK: kB3 and kB4.
    each_row(c, l, nk, [&](int k, int ik0) {
      const float v = row_sum(x.s(k, L.spec), ik0, nth);
      const float asum = v * dth;
      float dd = zero, pb2 = zero;
      if (asum > 1.E-8f) {
        dd = nka(k, kA2)[ik0] / asum;
        pb2 = nka(k, kA3)[ik0] / asum;
      }
      nka(k, kB3)[ik0] = dd;
      nka(k, kB4)[ik0] = pb2;
      nka(k, kBth0)[ik0] = pb2 > 0.001f ? 2.0f * p.ssdsbr : zero;
    });
    c.sync();
    each_bin(c, l, nspec, [&](int k, int i) {
      const int ik0 = x.row(i);
      const float a = x.s(k, L.spec)[i];
      const float pb = ((one - ssdsc[0]) * nka(k, kB4)[ik0]) * a + ssdsc[0] * zero;
      brl_of(k)[i] = pb / kTwoPiSq;
      const float dd = nka(k, kB3)[ik0];
      x.gs(k, L.vdds)[i] = dd;
      x.gs(k, L.vsds)[i] = dd * a;
    });
    c.sync();
  } else if (sdscase == 3) {
    // 1.b Mean-square slope (:2228-2254): per-IK direction sums, then the running sums over IK.
    const bool mss = ssdsc[7] > zero || ssdsc[10] > zero || ssdsc[17] > zero;
    if (mss) {
      each_row(c, l, nk, [&](int k, int ik0) {
        const float* const a = x.s(k, L.spec) + ik0 * nth;
        const float cg = x.s(k, L.cg1)[ik0];
        float mssp = zero, msspc2 = zero, mssps2 = zero;
        const float kp = dm::powf(x.s(k, L.wn1)[ik0], ssdsc[19]);
WWB_UNROLL(1)
        for (int ith = 0; ith < nth; ++ith) {
          const float msslong = ((kp * a[ith]) * f.dden[ik0]) / cg;
          msspc2 = msspc2 + msslong * f.ecos[ith];
          mssps2 = mssps2 + msslong * f.esin[ith];
          mssp = mssp + msslong;
        }
        nka(k, kB1)[ik0] = mssp;
        nka(k, kB2)[ik0] = msspc2;
        nka(k, kB3)[ik0] = mssps2;
      });
      c.sync();
      each_row(c, l, nk, [&](int k, int i0) {
        float m1 = zero, m3 = zero, m4 = zero;
WWB_UNROLL(1)
        for (int ik = 0; ik <= i0; ++ik) {
          m1 = m1 + nka(k, kB1)[ik];
          m3 = m3 + nka(k, kB2)[ik];
          m4 = m4 + nka(k, kB3)[ik];
        }
        nka(k, kMss1)[i0] = m1;
        float mssd = dm::atan2f(m4, m3);
        if (mssd < zero) mssd = mssd + kPi;
        nka(k, kMss2)[i0] = mssd;
      });
      c.sync();
    }
    // 2.c Romero 2019 (:2481-2520): what one IK gives, then its bins.
    each_row(c, l, nk, [&](int k, int ik0) {
      const SrceSh& s = x.sh[k];
      const int ik = ik0 + 1;
      const float* const a = x.s(k, L.spec) + ik0 * nth;
      const float t28 = 28.0f / ssdsc[15];
      const float ko = (kGrav / (s.r.ustar * s.r.ustar)) / (t28 * t28);
      const float kx = x.s(k, L.wn1)[ik0];
      const float kloc = dm::powf(kx, 2.0f - ssdsc[19]);
      const float k3 = (kx * kx) * kx;
      float dirforcum = s.r.dlwmean;
      if (ssdsc[10] > zero) dirforcum = nka(k, kMss2)[ik0];
      float sb = zero;
WWB_UNROLL(1)
      for (int ith = 0; ith < nth; ++ith)
        sb = sb + max_r((a[ith] * f.sig[ik]) * k3, .00000000000001f) * dth;
      nka(k, kBth0)[ik0] = sb;
      if (ssdsc[17] > zero) {
        float cd, sd;
        dm::sincosf(dirforcum, &sd, &cd);
        nka(k, kB1)[ik0] = cd;
        nka(k, kB2)[ik0] = sd;
        nka(k, kB3)[ik0] = dm::powf(nka(k, kMss1)[ik0] * kloc, ssdsc[13]);
      }
      nka(k, kB4)[ik0] = one + ssdsc[12] * dm::powf(max_r(kx / ko, one), ssdsc[14]);
      const float btover = sqrt_f(sb) - sqrt_f(p.ssdsbt);
      nka(k, kB5)[ik0] = btover;
      nka(k, kBrm12)[ik0] = ssdsc[1] * dm::powf(zero > btover ? zero : btover, 2.5f);
    });
    c.sync();
    each_bin(c, l, nspec, [&](int k, int i) {
      const int ik0 = x.row(i), ith = i - ik0 * nth, ik = ik0 + 1;
      const float kx = x.s(k, L.wn1)[ik0], a = x.s(k, L.spec)[i];
      const float k3 = (kx * kx) * kx;
      const float bthk = max_r((a * f.sig[ik]) * k3, .00000000000001f);
      const float cc = f.sig[ik] / kx;
      float lmod;
      if (ssdsc[17] > zero) {
        const float q = f.ecos[ith] * nka(k, kB1)[ik0] + f.esin[ith] * nka(k, kB2)[ik0];
        lmod = one + ssdsc[17] * (nka(k, kB3)[ik0] * (q * q));
        lmod = powf_i(lmod, ssdsc[18]);
      } else {
        lmod = one;
      }
      const float c9 = ssdsc[8], c13p1 = ssdsc[12] + one;
      float b = (((c9 * dm::expf(-(p.ssdsbr / bthk))) * nka(k, kB4)[ik0]) / c13p1) * lmod;
      const float xx = copysignf(b, nka(k, kB5)[ik0]);
      b = xx > zero ? xx : zero;
      brl_of(k)[i] = b;
      const float c2 = cc * cc;
      const float c5 = (cc * c2) * c2;
      const float sr = (((nka(k, kBrm12)[ik0] / kGrav2) * b) * c5) / f.sig[ik];
      x.gs(k, L.vsds)[i] = sr;
      x.gs(k, L.vdds)[i] = ((sr * p.ssdsbr) / max_r(bthk, 1.e-20f)) / max_r(a, 1e-20f);
    });
    c.sync();
  } else {
    each_bin(c, l, nspec, [&](int k, int i) {
      brl_of(k)[i] = x.gs(k, L.vsds)[i] = x.gs(k, L.vdds)[i] = zero;
    });
    each_row(c, l, nk, [&](int k, int ik0) {
      nka(k, kBth0)[ik0] = nka(k, kBrm12)[ik0] = zero;
    });
    c.sync();
  }

  // Whitecap parameters (:2581-2650), the per-IK part; the sums over IK stay in IK order (below).
  const bool wcap = x.sh[l.at(0)].in.flogrd57 || x.sh[l.at(0)].in.flogrd58;
  if (wcap) {
    const int fl = ffloor(p.aaircmin);
    const int ikc = fl < nk ? fl : nk;
    each_row(c, l, nk, [&](int k, int ik0) {
      const int ik = ik0 + 1;
      float c4 = zero, c5 = zero;
      if (ik <= ikc) {
        const float cc = f.sig[ik] / x.s(k, L.wn1)[ik0];
        const float cg = x.s(k, L.cg1)[ik0];
        const float v = row_sum(brl_of(k), ik0, nth);
        c4 = ((((((cc * cc) * v) * 2.0f) * kPi) / kGrav) * ssdsc[6]) * f.dden[ik0] /
             (f.sig[ik] * cg);
        const float pw = dm::powf(nka(k, kBrm12)[ik0] / ssdsc[1], 3.0f / 5.0f);
        const float* const b = brl_of(k) + ik0 * nth;
        float w = zero;
WWB_UNROLL(1)
        for (int i = 0; i < nth; ++i) w = w + (b[i] * (-ssdsc[1])) * pw;
        c5 = ((((cc * cc) * cc) * w) * p.aairgb / kGrav) * f.dden[ik0] / (f.sig[ik] * cg);
      }
      nka(k, kCoef4)[ik0] = c4;
      nka(k, kCoef5)[ik0] = c5;
    });
  }

  // Which blocks of four directions of a row the cumulative term has to sum: rows below the breaking
  // threshold are left out (:2558), and a block whose BRLAMBDA is zero adds +-0 to a sum that starts at
  // +0, which changes nothing while CUMULW is finite. Rows not made of whole blocks: one bit for all.
  const bool blocks = (nth & 3) == 0 && nth <= 128 && f.cum_finite;
  if (ssdsc[2] < zero) {
    each_row(c, l, nk, [&](int k, int ik0) {
      unsigned m = 0;
      if (nka(k, kBth0)[ik0] > p.ssdsbr) {
        if (blocks) {
          const float* const b = brl_of(k) + ik0 * nth;
WWB_UNROLL(1)
          for (int j = 0; j < nth; j += 4) {
            const F4 r = ld4(b + j);
            if (r.a != zero || r.b != zero || r.c != zero || r.d != zero) m |= 1u << (j >> 2);
          }
        } else {
          m = 1;
        }
      }
      reinterpret_cast<unsigned*>(nka(k, kA1))[ik0] = m;
    });
    c.sync();
  }

  // Wave-turbulence interaction and cumulative effect (:2533-2575).
  const bool turb = (ssdsc[2] != zero) || (ssdsc[4] != zero) || (ssdsc[20] != zero);
  if (turb && ssdsc[2] > zero) {
    // The isotropic form's sums over directions are one value per IK2, its sum over IK2 one per IK.
    each_row(c, l, nk, [&](int k, int ik0) { nka(k, kB1)[ik0] = row_sum(brl_of(k), ik0, nth); });
    c.sync();
    each_row(c, l, nk, [&](int k, int ik0) {
      const int ik = ik0 + 1;
      const float* const kk = x.s(k, L.wn1);
      const float cc = f.sig[ik] / kk[ik0];
      float ren = zero;
      if (ik > dikcumul)
WWB_UNROLL(1)
        for (int ik2 = ik1; ik2 <= ik - dikcumul; ++ik2) {
          const float cc2 = f.sig[ik2] / kk[ik2 - 1];
          const float cumulwiso = ((fabs_f(cc2 - cc) * f.dsip[ik2]) / (cc2 * 0.5f)) * dth;
          ren = ren - cumulwiso * nka(k, kB1)[ik2 - 1];
        }
      nka(k, kRen)[ik0] = ren;
    });
    c.sync();
  }
  if (turb) {
WWB_UNROLL(1)
    for (int j = 0; j < l.n; j += kTogether) {
      one_copy();
      const SlotList g = l.part(j, kTogether);
      if (g.n == 1) sds4_turb<1>(c, x, g, blocks, dikcumul, ik1, R + kA1 * K, R + kRen * K);
      else sds4_turb<kTogether>(c, x, g, blocks, dikcumul, ik1, R + kA1 * K, R + kRen * K);
    }
  }
  c.sync();
  if (wcap) {
    const int fl = ffloor(p.aaircmin);
    const int ikc = fl < nk ? fl : nk;
    each_chain(c, 1, l, [&](int k) {
      SrceSh& s = x.sh[k];
      const float* const coef4 = nka(k, kCoef4);
      const float* const coef5 = nka(k, kCoef5);
      const float* const mftk = x.s(k, L.mft);
      float wc0 = zero, wc1 = zero, wc3 = zero;
      if (s.in.flogrd57) {
WWB_UNROLL(1)
        for (int ik = ik1; ik <= ikc; ++ik) {
          wc0 = wc0 + coef4[ik - 1] * (one - wc0);
          wc3 = wc3 + coef5[ik - 1];
        }
      }
      if (s.in.flogrd58) {
WWB_UNROLL(1)
        for (int ik = ik1; ik <= nk; ++ik) wc1 = wc1 + coef4[ik - 1] * mftk[ik - 1];
      }
      s.whitecap[0] = wc0;
      s.whitecap[1] = wc1;
      s.whitecap[2] = zero;
      s.whitecap[3] = wc3;
    });
  }
}

// --------------------------------------------------------------------------------- the step
/// Waits for the tail warp if it was given work.
WWB_PD void tail_done(const Grp& c, bool& tail) {
  if (tail) c.tail_wait();
  tail = false;
}

/// A step up to the update (:1210-1847) of the listed slots: the step count, W3SLN1, the DIA, W3SDS4,
/// W3SDB1, W3SBT1, the time step, the new spectrum and the terms of the closing sums.
template <class G>
WWB_PD void srce_advance(const Grp& c, const G& x, const SlotList& l, bool& tail) {
  const srce::Params& p = *x.p;
  const SrceLayout& L = *x.L;
  const int nk = L.nk, nth = x.nth(), nspec = L.nspec;
  const int R = (nspec + 3) & ~3;
  if (p.ln1) {
    // W3SLN1 (w3sln1md.F90:56-211): VSLN = WNF(IK) * DIRF(ITH), formed where it is read.
    auto fmin2 = [](float a, float b) { return (b < a) ? b : a; };
    auto fmax2 = [](float a, float b) { return (b > a) ? b : a; };
    each_row(c, l, nth, [&](int k, int ith) {
      const float m =
          fmax2(0.0f, x.g->ecos[ith] * x.sh[k].cosw + x.g->esin[ith] * x.sh[k].sinw);
      const float m2 = m * m;
      x.s(k, L.dirf)[ith] = m2 * m2;
    });
    each_row(c, l, nk, [&](int k, int ik) {
      const SrceSh& s = x.sh[k];
      const float ustar = s.r.ustar;
      const float u2 = ustar * ustar;
      const float fac = p.slnc1 * (u2 * u2);
      const float ff1 = p.fspm * kGrav / (28.0f * ustar);
      const float ff2 = p.fshf * fmin2(x.g->sig[nk - 1], s.fhigh);
      const float ffilt = fmin2(2.0f * x.g->sig[nk - 1], fmax2(ff2, ff1));
      const float rfr = x.g->sig[ik] / ffilt;
      float v = 0.0f;
      if (!(rfr < 0.5f)) {
        const float r2 = rfr * rfr;
        const float rm4 = 1.0f / (r2 * r2);
        v = fac / x.s(k, L.wn1)[ik] * dm::expf(-rm4);
      }
      x.s(k, L.wnf)[ik] = v;
    });
  }
  srce_dia(c, x, l);
  srce_sds4(c, x, l);
  // W3SDB1 (:1321).
  each_chain(c, 0, l, [&](int k) {
    SrceSh& s = x.sh[k];
    const float emean = s.r.emean;
    const bool early = static_cast<double>(emean) < 0x1p-1022;
    s.early = early ? 1 : 0;
    if (!early) {
      const double thr = static_cast<double>(0x1p-126f);
      double hm;
      if (p.fdonly != 0) {
        hm = static_cast<double>(p.sdbc2) * static_cast<double>(s.depth);
      } else {
        const float dpos = (s.depth > 0.0f) ? s.depth : 0.0f;
        const double wnm = static_cast<double>(s.r.wnmean);
        hm = static_cast<double>(p.sdbc2) / wnm * dm::tanh_d(wnm * static_cast<double>(dpos));
      }
      const double hrms = sqrt(8. * static_cast<double>(emean));
      double bb, b;
      if (hm > thr) {
        bb = hrms * hrms / (hm * hm);
        b = sqrt(bb);
      } else {
        bb = 0.;
        b = 0.;
      }
      double q0 = 0.;
      if (b <= 0.5) {
        q0 = 0.;
      } else if (b <= 1.) {
        const double t = 2. * b - 1.;
        q0 = t * t;
      }
      double qb;
      if (b <= 0.2) {
        qb = 0.;
      } else if (b < 1.) {
        const double arg = dm::exp_d((q0 - 1.) / bb);
        qb = q0 - bb * (q0 - arg) / (bb - arg);
WWB_UNROLL(1)
        for (int is = 1; is <= 3; ++is) qb = dm::exp_d((qb - 1.) / bb);
      } else {
        qb = static_cast<double>(1.0f - 0x1p-126f);
      }
      double cbj = 0.;
      if (b != 1. && (bb > thr) && (fabs(bb - qb) > thr)) {
        if (bb < 1.0) {
          cbj = 2. * static_cast<double>(p.sdbc1) * qb * static_cast<double>(s.r.fmean) / bb;
        } else {
          cbj = 2. * static_cast<double>(p.sdbc1) * static_cast<double>(s.r.fmean) * bb;
        }
      }
      s.vddb = static_cast<float>(-cbj);
    }
  });
  // The time-step limits (:1427-1437).
  each_chain(c, 2, l, [&](int k) {
    SrceSh& s = x.sh[k];
    s.nsteps = s.nsteps + 1;
    s.nkh = min_i(nk, fint(p.facti1 * dm::logf(mx(1.E-7f, s.fhigh)) + p.facti2));
    s.nkh1 = min_i(nk, s.nkh + 1);
    s.nspech = s.nkh1 * nth;
    s.afilt = mx(x.s(k, L.dam)[nk - 1], p.xflt * s.r.amax);
    s.vmin = 0x7f800000u;
  });
  c.sync();
  // :1484-1533, VS, VD and the MIN over IS of the time step's limit.
  {
    struct Slot {
      const float *spec, *vdin, *vsnl, *vdnl, *specinit, *wnf, *dirf, *cbeta, *dam;
      float *vsds, *vdds;
      int nspech, nscut, k;
      bool ice;
      float iln, iin, inl, ids, afilt;
      unsigned low;  ///< bits of the smallest limit so far
    };
    struct In {
      float vdin, vsnl, vdnl, vsds, vdds, specinit;
    };
    // The limits are never negative and never NaN (mx and mn take their second operand for
    // one), so their order is that of their bits.
    bins_ld<2>(c, l, nspec, [&](int k) {
      const SrceSh& s = x.sh[k];
      return Slot{x.s(k, L.spec), x.gs(k, L.vdin), x.gs(k, L.vsnl), x.gs(k, L.vdnl),
                  x.gs(k, L.specinit), x.s(k, L.wnf), x.s(k, L.dirf), x.s(k, L.cbeta), x.s(k, L.dam),
                  x.gs(k, L.vsds), x.gs(k, L.vdds), s.nspech, s.nscut, k, s.in.inflags24 != 0,
                  s.icescaleln, s.icescalein, s.icescalenl, s.icescaleds, s.afilt, 0x7f800000u};
    }, [&](const Slot& s, int i) {
      return In{s.vdin[i], s.vsnl[i], s.vdnl[i], s.vsds[i], s.vdds[i], s.specinit[i]};
    }, [&](Slot& s, int i, const In& in) {
      if (i >= s.nspech) return;
      const int ik = x.row(i);
      const float spec = s.spec[i];
      float vdin = in.vdin;
      float vsin = vdin * spec;
      float vsnl = in.vsnl, vdnl = in.vdnl, vsds = in.vsds, vdds = in.vdds;
      float vsln = p.ln1 ? s.wnf[ik] * s.dirf[i - ik * nth] : 0.0f;
      float vdbt = 0.0f, vsbt = 0.0f;
      if (s.nscut >= 0) {
        vdbt = i < s.nscut ? s.cbeta[x.g->mapwn[i] - 1] : 0.0f;
        vsbt = vdbt * spec;
      }
      if (s.ice) {
        vsnl = s.inl * vsnl;
        vdnl = s.inl * vdnl;
        vsln = s.iln * vsln;
        vsin = s.iin * vsin;
        vdin = s.iin * vdin;
        vsds = s.ids * vsds;
        vdds = s.ids * vdds;
      }
      const float vs = (((vsln + vsin) + vsnl) + vsds) + vsbt;
      const float vd = ((vdin + vdnl) + vdds) + vdbt;
      s.vsds[i] = vs;
      s.vdds[i] = vd;
      const float damax = mn(mx(p.xrel * in.specinit, s.afilt), s.dam[ik]);
      const float afac = 1.0f / mx(fabs_f(vs / damax), 1.E-10f);
      const unsigned v = dm::asuint(afac / mx(mn(vd, 0.0f) * afac + 1.0f, 1.E-10f));
      s.low = v < s.low ? v : s.low;
    }, [&](const Slot& s) {
#if defined(__CUDA_ARCH__)
      const unsigned m = __reduce_min_sync(0xffffffffu, s.low);
      if (c.lane() == 0) atomicMin(&x.sh[s.k].vmin, m);
#else
      if (s.low < x.sh[s.k].vmin) x.sh[s.k].vmin = s.low;
#endif
    });
  }
  c.sync();
  tail_done(c, tail);
  each_chain(c, 0, l, [&](int k) {
    SrceSh& s = x.sh[k];
    const float dtg = s.in.dtg;
    float dt = mn(mn(p.dtmax, dtg - s.dttot), dm::asfloat(s.vmin));
    dt = mx(dt, 0.5f);
    s.dtdyn = s.dtdyn + dt;
    const float rest = dtg - s.dttot;
    const int idt = 1 + fint((rest * 0.99f) / dt);
    dt = rest / static_cast<float>(idt);
    const bool shave = dt < p.dtmin && dt < rest;
    s.shave = shave ? 1 : 0;
    dt = mx(mn(p.dtmin, rest), dt);
    s.dt = dt;
    s.dttot = s.dttot + dt;
    s.tauwix = s.tauwix + (s.tauwx * s.drat) * dt;
    s.tauwiy = s.tauwiy + (s.tauwy * s.drat) * dt;
    s.tauwnx = s.tauwnx + (s.drat * s.tauwax) * dt;
    s.tauwny = s.tauwny + (s.drat * s.tauway) * dt;
  });
  c.sync();
  // :1761-1847, the update and the terms of the ordered sums (PHIAW and PHIBBL's terms, and whether a
  // bin counts for the wind sea's height).
  {
    struct Slot {
      float *spec, *vsdb, *t, *tb;
      const float *vdin, *vs, *vd, *cbeta, *cg, *dam;
      unsigned char* wind;
      int nspech, nscut;
      bool ice, early, shave;
      float iin, dt, vddb;
    };
    struct In {
      float vdin, vs, vd;
    };
    bins_ld<2>(c, l, nspec, [&](int k) {
      const SrceSh& s = x.sh[k];
      float* const t = x.tr(k);
      return Slot{x.s(k, L.spec), x.gs(k, L.vsdb), t, t + R, x.gs(k, L.vdin), x.gs(k, L.vsds),
                  x.gs(k, L.vdds), x.s(k, L.cbeta), x.s(k, L.cg1), x.s(k, L.dam),
                  reinterpret_cast<unsigned char*>(t + 2 * R), s.nspech, s.nscut,
                  s.in.inflags24 != 0, s.early != 0, s.shave != 0, s.icescalein, s.dt, s.vddb};
    }, [&](const Slot& s, int i) { return In{s.vdin[i], s.vs[i], s.vd[i]}; },
    [&](const Slot& s, int i, const In& in) {
      const int ik = x.row(i);
      const float dt = s.dt, hdt = dt;
      const float spec = s.spec[i];
      const bool low = i < s.nspech;
      float vdin = in.vdin;
      float vsin = vdin * spec;
      if (s.ice && low) {
        vsin = s.iin * vsin;
        vdin = s.iin * vdin;
      }
      float vsdb;
      if (s.early) {
        vsdb = s.vsdb[i];
      } else {
        vsdb = s.vddb * spec;
        s.vsdb[i] = vsdb;
      }
      float vdbt = 0.0f, vsbt = 0.0f;
      if (s.nscut >= 0) {
        vdbt = i < s.nscut ? s.cbeta[x.g->mapwn[i] - 1] : 0.0f;
        vsbt = vdbt * spec;
      }
      if (low) {
        const float einc1 = (dt * in.vs) / mx(1.0f - hdt * in.vd, 1.0f);
        float v;
        if (s.shave) {
          const float einc2 = copysignf(mn(fabs_f(einc1), s.dam[ik]), einc1);
          v = mx(spec + einc2, 0.0f);
        } else {
          v = mx(spec + einc1, 0.0f);
        }
        const float e2 = (dt * vsdb) / mx(1.0f - hdt * s.vddb, 1.0f);
        s.spec[i] = mx(v + e2, 0.0f);
      }
      const float factor = x.g->dden[ik] / s.cg[ik];
      s.t[i] = ((vsin * dt) * factor) / mx(1.0f - vdin * dt, 1.0f);
      s.tb[i] = -(((vsbt * dt) * factor) / mx(1.0f - vdbt * dt, 1.0f));
      s.wind[i] = vsin > 0.0f ? 1 : 0;
    }, [](const Slot&) {});
  }
  c.sync();
}

/// The closing sums' chains (:1815-1847), roles 4-6.
template <class G>
WWB_PD void srce_sums(const Grp& c, const G& x, const SlotList& l) {
  const SrceLayout& L = *x.L;
  const int R = (L.nspec + 3) & ~3;
  each_chain_of(c, 4, 2, l, [&](int r, int k) {
    float* const to = r ? &x.sh[k].phibbl : &x.sh[k].phiaw;
    *to = sum4(x.tr(k) + r * R, L.nspec, *to);  // PHIBBL's terms are stored negated
  });
  each_chain(c, 6, l, [&](int k) {
    // A bin without wind input adds -0, which changes nothing.
    const float* const sp = x.s(k, L.spec);
    const unsigned char* const wind = reinterpret_cast<const unsigned char*>(x.tr(k) + 2 * R);
    float v = 0.0f;
WWB_UNROLL(1)
    for (int ik = 0; ik < L.nk; ++ik) {
      const float factor = x.g->dden[ik] / x.s(k, L.cg1)[ik];
      const int nth = x.nth();
      int i = ik * nth;
      const int end = i + nth;
      if ((nth & 3) == 0) {
WWB_UNROLL(3)
        for (; i < end; i += 4) {
          const F4 q = ld4(sp + i);
          const uint32_t b = *reinterpret_cast<const uint32_t*>(wind + i);
          const float t0 = q.a * factor, t1 = q.b * factor, t2 = q.c * factor, t3 = q.d * factor;
          v = v + (b & 0xffu ? t0 : -0.0f);
          v = v + (b & 0xff00u ? t1 : -0.0f);
          v = v + (b & 0xff0000u ? t2 : -0.0f);
          v = v + (b & 0xff000000u ? t3 : -0.0f);
        }
      }
WWB_UNROLL(1)
      for (; i < end; ++i) {
        const float t = sp[i] * factor;
        v = v + (wind[i] ? t : -0.0f);
      }
    }
    x.sh[k].whitecap[2] = sqrt_f(v) * 4.0f;
  });
}

/// After the step's W3SPR4 (:1880-1997): FHIGH, MLIM, SEED, the tail for running slots; SPECINIT and
/// FHIGH's first value for the slots that end their initialisation (:1122-1179).
template <class G>
WWB_PD void srce_shape(const Grp& c, const G& x, const SlotList& run,
                       const SlotList& fresh2) {
  const srce::Params& p = *x.p;
  const SrceLayout& L = *x.L;
  const int nk = L.nk, nth = x.nth(), nspec = L.nspec;
  each_chain(c, 0, run, [&](int k) {
    SrceSh& s = x.sh[k];
    s.fage = p.ffxfa * dm::tanhf((((s.in.u10abs * 0.3f) * s.r.fmeanws) * kTpi) / kGrav);
    const float fh1 = (p.ffxfm + s.fage) * s.r.fmean1;
    const float fh2 = p.ffxpm / s.r.ustar;
    s.fhigh = mn(mx(fh1, fh2), x.g->sig[nk - 1]);
    s.nkh = max_i(min_i(s.nkh1, fint(p.facti1 * dm::logf(mx(1.E-7f, s.fhigh)) + p.facti2)), 2);
    s.mlim = -1.0f;
    if (s.dttot >= s.in.dtg * 0.9999f) {
      const float hm = (p.fhmax * dm::tanhf(mx(0.0f, s.in.d_inp) * s.r.wnmean)) /
                       mx(s.r.wnmean, 9.99999974737875163555145263671875e-5f);
      const float em = (hm * hm) * 6.25e-2f;
      if (s.r.emean > em && s.r.emean > 1.E-30f) {
        s.mlim = em;  // MLIM applies with EM
      }
    }
    s.done = (s.dttot >= 0.9999f * s.in.dtg || s.nsteps >= 100000) ? 1 : 0;
  });
  each_chain(c, 1, fresh2, [&](int k) {
    SrceSh& s = x.sh[k];
    s.tws = 1.0f / s.r.fmeanws;
    s.fage = 0.0f;
    s.fhigh = mx((p.ffxfm + 0.0f) * mx(s.r.fmeanws, s.r.fmean1), p.ffxpm / s.r.ustar);
    s.done = 0;
  });
  each_bin(c, fresh2, nspec,
           [&](int k, int i) { x.gs(k, L.specinit)[i] = x.s(k, L.spec)[i]; });
  c.sync();
  if (run.n == 0) return;
  SlotList lim{};
WWB_UNROLL(1)
  for (int j = 0; j < run.n; ++j)
    if (x.sh[run.at(j)].mlim >= 0.0f) lim.add(run.at(j));
  if (lim.n) {
    each_bin(c, lim, nspec, [&](int k, int i) {
      float* const sp = x.s(k, L.spec) + i;
      *sp = x.sh[k].mlim * (*sp / x.sh[k].r.emean);
    });
    c.sync();
    each_chain(c, 0, lim, [&](int k) { x.sh[k].r.emean = x.sh[k].mlim; });
  }
  if (p.seed) {
    each_bin(c, run, nspec, [&](int k, int i) {
      const SrceSh& s = x.sh[k];
      const int ik = x.row(i) + 1;
      if (ik >= min_i(nk, s.nkh)) {
        const int ith = i - (ik - 1) * nth;
        const float uc = (p.facsd * kGrav) / x.g->sig[ik - 1];
        const float w = x.s(k, L.wn1)[ik - 1];
        float slev = ((mn(mx(s.in.u10abs / uc - 1.0f, 0.0f), 1.0f) * 6.25E-4F) / ((w * w) * w)) /
                     x.g->sig[ik - 1];
        if (s.in.inflags24) slev = (1.0f - s.in.ice) * slev;
        float sn, cs;
        dm::sincosf(s.in.u10dir - x.f->th[ith], &sn, &cs);
        const float cc = mx(cs, 0.0f);
        float* const sp = x.s(k, L.spec) + i;
        *sp = mx(slev * (cc * cc), *sp);
      }
    });
    c.sync();
  }
  // :1985-1997, the tail: a recurrence up the frequencies, parallel over directions.
  each_row(c, run, nth, [&](int k, int ith) {
    const int nkh = x.sh[k].nkh;
    if (nkh >= nk) return;
    float* const sp = x.s(k, L.spec) + ith;
    float v = sp[(nkh - 1) * nth];
WWB_UNROLL(1)
    for (int ik = nkh; ik < nk; ++ik) {
      v = v * p.fachfa + 0.0f;
      sp[ik * nth] = v;
    }
  });
  c.sync();
}

/// 3. After the loop (:2050-2350), FLD2 excepted (ww_srce_init refuses it).
template <class G>
WWB_PD void srce_finish(const Grp& c, const G& x, const SlotList& l) {
  const srce::Params& p = *x.p;
  const SrceLayout& L = *x.L;
  const int nk = L.nk, nth = x.nth(), nspec = L.nspec;
  // Per-IK band sums: eband, a1band, b1band.
  each_row(c, l, nk, [&](int k, int ik) {
    const float* const spec = x.s(k, L.spec);
    const float* const specinit = x.gs(k, L.specinit);
    float eband = 0.0f, a1band = 0.0f, b1band = 0.0f;
WWB_UNROLL(1)
    for (int ith = 0; ith < nth; ++ith) {
      const float diff = specinit[ith + ik * nth] - spec[ith + ik * nth];
      eband = diff + eband;
      a1band = x.g->ecos[ith] * diff + a1band;
      b1band = x.g->esin[ith] * diff + b1band;
    }
    float* const T = x.tr(k);
    T[3 * ik] = eband;
    T[3 * ik + 1] = a1band;
    T[3 * ik + 2] = b1band;
  });
  c.sync();
  each_chain(c, 0, l, [&](int k) {
    SrceSh& s = x.sh[k];
    const float* const T = x.tr(k);
    const float* const spec = x.s(k, L.spec);
    s.dtdyn = s.dtdyn / static_cast<float>(max_i(s.nsteps, 1));
    s.fcut = s.fhigh * kTpiInv;
    float efinish = 0.0f, mwxfinish = 0.0f, mwyfinish = 0.0f;
WWB_UNROLL(1)
    for (int ik = 0; ik < nk; ++ik) {
      const float dden = x.g->dden[ik], cg = x.s(k, L.cg1)[ik], wn = x.s(k, L.wn1)[ik];
      efinish = (dden * T[3 * ik]) / cg + efinish;
      mwxfinish = (((dden * T[3 * ik + 1]) / cg) * wn) / x.g->sig[ik] + mwxfinish;
      mwyfinish = (wn * ((dden * T[3 * ik + 2]) / cg)) / x.g->sig[ik] + mwyfinish;
    }
    const float dtg = s.in.dtg;
    s.tauox = ((s.tauwix + mwxfinish * kGrav) - s.taubbl[0]) / dtg;
    s.tauoy = ((s.tauwiy + mwyfinish * kGrav) - s.taubbl[1]) / dtg;
    s.tauwix = s.tauwix / dtg;
    s.tauwiy = s.tauwiy / dtg;
    s.tauwnx = s.tauwnx / dtg;
    s.tauwny = s.tauwny / dtg;
    s.taubbl[0] = s.taubbl[0] / dtg;
    s.taubbl[1] = s.taubbl[1] / dtg;
    float cc, sn;
    dm::sincosf(s.r.usdir, &sn, &cc);
    const float q = s.r.ustar * (s.r.ustar * (s.in.coef * (s.in.dair * s.in.coef)));
    s.tauocx = q * cc + (s.tauox - s.tauwix) * kDwat;
    s.tauocy = q * sn + (s.tauoy - s.tauwiy) * kDwat;
    const float dg = kDwat * kGrav;
    s.phioc = (((s.phiaw + efinish) - s.phibbl) * dg) / dtg;
    s.phiaw = (s.phiaw * dg) / dtg;
    s.phibbl = (s.phibbl * dg) / dtg;
    // The ice block without dispersion (:2124-2259): ATT = 1, SPEC unchanged; the sums are of
    // zeros and kept for their signed zeros.
    if (s.in.inflags24 && s.in.ice > 0.0f && !p.ic_numerics) {
      s.tauice[0] = s.tauice[1] = 0.0f;
      s.phice = 0.0f;
WWB_UNROLL(1)
      for (int ik = 0; ik < nk; ++ik) {
        const float factor = x.g->dden[ik] / x.s(k, L.cg1)[ik];
        const float factor2 = ((factor * kGrav) * x.s(k, L.wn1)[ik]) / x.g->sig[ik];
WWB_UNROLL(1)
        for (int ith = 0; ith < nth; ++ith) {
          const int is = ith + ik * nth;
          const float sp2 = spec[is];
          const float spn = static_cast<float>(1.0 * static_cast<double>(sp2));
          s.phice = s.phice + (spn - sp2) * factor;
          s.tauice[0] = s.tauice[0] - ((spn - sp2) * factor2) * x.g->ecos[is];
          s.tauice[1] = s.tauice[1] - ((spn - sp2) * factor2) * x.g->esin[is];
        }
      }
      s.phice = (((-1.0f * kDwat) * kGrav) * s.phice) / dtg;
      s.tauice[0] = s.tauice[0] / dtg;
      s.tauice[1] = s.tauice[1] / dtg;
    }
  });
  c.sync();
  const int nlast = (nspec % 4 == 3) ? nspec - 1 : nspec;
  each_bin(c, l, nspec, [&](int k, int i) {
    float* const sp = x.s(k, L.spec) + i;
    const float v = x.sh[k].in.it == 0 ? x.gs(k, L.specinit)[i] : *sp;
    *sp = i < nlast ? mx(v, 0.0f) : mx(0.0f, v);
  });
  c.sync();
}

/// The step's flags and a point's PIN packet (ww_kokkos_c.hpp:231-240).
WWB_PD SrceIn srce_in(int it, int inflags24, int flogrd57, int flogrd58, float dtg,
                      const float* pin) {
  SrceIn in{};
  in.it = it;
  in.inflags24 = inflags24;
  in.flogrd57 = flogrd57;
  in.flogrd58 = flogrd58;
  in.dtg = dtg;
  in.d_inp = pin[srce::IN_D_INP];
  in.u10abs = pin[srce::IN_U10ABS];
  in.u10dir = pin[srce::IN_U10DIR];
  in.as = pin[srce::IN_AS];
  in.ice = pin[srce::IN_ICE];
  in.dair = pin[srce::IN_DAIR];
  in.coef = pin[srce::IN_COEF];
  return in;
}

/// A point's INOUT scalars (PSC packet, WHITECAP, TAUBBL, TAUICE) into the shared state, and
/// back with SHAVE (single thread).
WWB_PD void srce_psc_in(SrceSh& s, const float* psc, const float* wc, const float* tb,
                        const float* ti) {
  s.r.ustar = psc[srce::SC_USTAR];
  s.r.usdir = psc[srce::SC_USTDIR];
  s.tauwx = psc[srce::SC_TAUWX];
  s.tauwy = psc[srce::SC_TAUWY];
  s.dtdyn = psc[srce::SC_DTDYN];
  s.fcut = psc[srce::SC_FCUT];
  s.tauox = psc[srce::SC_TAUOX];
  s.tauoy = psc[srce::SC_TAUOY];
  s.tauwix = psc[srce::SC_TAUWIX];
  s.tauwiy = psc[srce::SC_TAUWIY];
  s.tauwnx = psc[srce::SC_TAUWNX];
  s.tauwny = psc[srce::SC_TAUWNY];
  s.phiaw = psc[srce::SC_PHIAW];
  s.r.charn = psc[srce::SC_CHARN];
  s.tws = psc[srce::SC_TWS];
  s.phioc = psc[srce::SC_PHIOC];
  s.phibbl = psc[srce::SC_PHIBBL];
  s.phice = psc[srce::SC_PHICE];
  s.tauocx = psc[srce::SC_TAUOCX];
  s.tauocy = psc[srce::SC_TAUOCY];
  s.r.wnmean = psc[srce::SC_WNMEAN];
  s.fpi = psc[srce::SC_FPI];
  for (int j = 0; j < 4; ++j) s.whitecap[j] = wc[j];
  s.taubbl[0] = tb[0];
  s.taubbl[1] = tb[1];
  s.tauice[0] = ti[0];
  s.tauice[1] = ti[1];
  s.shave = 0;
}

WWB_PD void srce_psc_out(const SrceSh& s, float* psc, float* wc, float* tb, float* ti,
                         int* shave) {
  psc[srce::SC_USTAR] = s.r.ustar;
  psc[srce::SC_USTDIR] = s.r.usdir;
  psc[srce::SC_TAUWX] = s.tauwx;
  psc[srce::SC_TAUWY] = s.tauwy;
  psc[srce::SC_DTDYN] = s.dtdyn;
  psc[srce::SC_FCUT] = s.fcut;
  psc[srce::SC_TAUOX] = s.tauox;
  psc[srce::SC_TAUOY] = s.tauoy;
  psc[srce::SC_TAUWIX] = s.tauwix;
  psc[srce::SC_TAUWIY] = s.tauwiy;
  psc[srce::SC_TAUWNX] = s.tauwnx;
  psc[srce::SC_TAUWNY] = s.tauwny;
  psc[srce::SC_PHIAW] = s.phiaw;
  psc[srce::SC_CHARN] = s.r.charn;
  psc[srce::SC_TWS] = s.tws;
  psc[srce::SC_PHIOC] = s.phioc;
  psc[srce::SC_PHIBBL] = s.phibbl;
  psc[srce::SC_PHICE] = s.phice;
  psc[srce::SC_TAUOCX] = s.tauocx;
  psc[srce::SC_TAUOCY] = s.tauocy;
  psc[srce::SC_WNMEAN] = s.r.wnmean;
  psc[srce::SC_FPI] = s.fpi;
  for (int j = 0; j < 4; ++j) wc[j] = s.whitecap[j];
  tb[0] = s.taubbl[0];
  tb[1] = s.taubbl[1];
  ti[0] = s.tauice[0];
  ti[1] = s.tauice[1];
  *shave = s.shave;
}

/// W3SRCE for the points `src` hands out: slots are loaded, taken through their states and stored
/// until there is nothing left to load and every slot is empty.
///   src.load(c, x, fresh): fills empty slots (SPEC, WN1, CG1, the packets, the state) and lists them
///   src.store(c, x, done): writes the finished slots' results out
/// Both are called by the whole CTA and end with a barrier.
template <class G, class Src>
WWB_PD void srce_run(const Grp& c, const G& x, Src& src) {
  const SrceLayout& L = *x.L;
  const int R = (L.nspec + 3) & ~3;
  const int spr4_off = 2 * R + ((((R + 3) / 4) + 3) & ~3);
  const bool sin4_at_init = x.q->sintailpar[3] > 0.5f;  // :1100
  const bool spr4_twice = x.q->sintailpar[3] < 0.5f;    // :2012
  srce_common(c, x);
  bool tail = false;  // the tail warp is at work
  for (;;) {
    SlotList fresh{};
    src.load(c, x, fresh);
    if (fresh.n) srce_begin(c, x, fresh);
    SlotList all{}, run{}, fresh2{}, wind{}, done{};
WWB_UNROLL(1)
    for (int k = 0; k < x.ns; ++k) {
      const int st = x.sh[k].state;
      if (st == kIdle) continue;
      all.add(k);
      if (st == kRun) run.add(k);
      if (st == kFresh2) fresh2.add(k);
      if (st != kFresh1 || sin4_at_init) wind.add(k);
    }
    if (all.n == 0) break;
    if (run.n) srce_advance(c, x, run, tail);
    // W3SPR4, what follows it, W3SIN4; for SINTAILPAR(4) < 0.5 running slots take W3SPR4 and (unless
    // they end) the next step's W3SIN4 once more. Otherwise the next step's W3SIN4 is this one: it
    // reads the same spectrum, USTAR, Z0 and wind, so it gives the same bits.
WWB_UNROLL(1)
    for (int rep = 0;; ++rep) {
      const SlotList& spr = rep == 0 ? all : run;
      spr4_sums(c, x, spr, spr4_off);
      c.sync();
      tail_done(c, tail);
      spr4_chains(c, x, spr, spr4_off);
      if (rep == 0 && run.n) srce_sums(c, x, run);
      c.sync();
      each_chain(c, 2, spr, [&](int k) {
        SrceSh& s = x.sh[k];
        s.r.dlwmean = dm::atan2f(s.chains[1], s.chains[0]);
        s.r.amax = s.chains[2];
      });
      if (rep == 0) {
        srce_shape(c, x, run, fresh2);
WWB_UNROLL(1)
        for (int j = 0; j < run.n; ++j)
          if (x.sh[run.at(j)].done) done.add(run.at(j));
      }
      SlotList next = wind;
      if (rep == 1) {
        next = SlotList{};
WWB_UNROLL(1)
        for (int j = 0; j < run.n; ++j)
          if (!x.sh[run.at(j)].done) next.add(run.at(j));
        c.sync();
      }
      if (next.n) {
        srce_sin4(c, x, next);
        tail = x.box != nullptr;
      }
      if (!(rep == 0 && spr4_twice && run.n)) break;
    }
    each_chain(c, 0, all, [&](int k) {
      const int st = x.sh[k].state;
      x.sh[k].state = st == kFresh1 ? kFresh2 : kRun;
    });
    c.sync();
    if (done.n) {
      tail_done(c, tail);
      srce_finish(c, x, done);
      src.store(c, x, done);
    }
  }
}

/// One point's context as a caller without a work queue holds it: configuration, tables, inputs, the
/// working set of one slot with SPEC, WN1, CG1 and the packets in place.
struct SrceCtx {
  const srce::Params* p;
  const SrceGrid* g;
  const st4::Params* q;
  const Fields* f;
  const Snl1Dev* n;
  SrceIn in;
  float* w;   ///< the shared part of the working set (SrceLayout)
  float* gw;  ///< the global part
  const SrceLayout* L;
  SrceSh* sh;
};

struct OnePoint {
  SrceIn in;
  bool taken = false;
  WWB_PD void load(const Grp&, const SrceGroup<0>& x, SlotList& fresh) {
    if (taken) return;
    taken = true;
    x.sh[0].in = in;
    x.sh[0].state = in.it != 0 ? kFresh1 : kFresh2;
    fresh.add(0);
  }
  WWB_PD void store(const Grp&, const SrceGroup<0>& x, const SlotList&) { x.sh[0].state = kIdle; }
};

/// W3SRCE for one point by one thread (the host build).
inline void srce_point(const Cta&, const SrceCtx& x) {
  const Grp c{0, 1};
  const SrceGroup<0> g{x.p, x.g, x.q, x.f, x.n, x.L, x.w, x.gw, x.w + x.L->common + x.L->ws, x.sh, 1, nullptr};
  OnePoint src{x.in};
  srce_run(c, g, src);
}

}  // namespace pt
}  // namespace wwb
