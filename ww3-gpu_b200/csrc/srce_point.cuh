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
// instruction cache: 36 x 36 bins, 9,520 points took 419 ms, 27.7 ms for a launch of 5 points.
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

/// Points a CTA integrates side by side.
constexpr int kSlots = 4;

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
  // W3SIN4
  float uorb, pturb, pvisc, fw, fu, fud, ustarsigma, const1;
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
  int pwsig, pwdir, tail, common;
  int ws, spec, llws, wn1, cg1, dam, pwwn, mft, cbeta, wnf, dirf;
  int tslot;           ///< transient floats a slot needs outside the DIA
  int dia;             ///< transient floats of one slot's DIA
  // global scratch per slot
  int specinit, vdin, vsnl, vdnl, vsds, vdds, vsdb, da, alen, work0, work1;
  int total_s;         ///< floats of shared memory with one slot
  int total_g;         ///< floats of global scratch per slot
};

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
  L.tail = o; o += r4(6 * kJtot);
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
  L.ws = o - L.common;
  while (L.ws % 32 != 4) L.ws += 4;
  L.tslot = 2 * R + r4((R + 3) / 4) + 8 * K;                  // closing sums + W3SPR4
  if (R + kNkWork * K > L.tslot) L.tslot = R + kNkWork * K;     // W3SDS4
  const int sin4 = R + r4((R + 3) / 4) + 9 * K;
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
  L.work0 = g;
  L.work1 = g + R;
  const int d = 4 * r4(L.alen) + R;
  g += d > 2 * R ? d : 2 * R;
  L.total_g = (g + 31) & ~31;
  L.total_s = srce_shared_floats(L, 1);
  return L;
}

/// A CTA of warps (on the host: one warp of one lane).
struct Grp {
  int tid, nthr;
  WWB_PD void sync() const {
#if defined(__CUDA_ARCH__)
    __syncthreads();
#endif
  }
  WWB_PD void syncwarp() const {
#if defined(__CUDA_ARCH__)
    __syncwarp();
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

/// Up to kSlots slot numbers, in registers.
struct SlotList {
  int n = 0;
  unsigned ids = 0;
  WWB_PD void add(int k) {
    ids |= static_cast<unsigned>(k) << (4 * n);
    ++n;
  }
  WWB_PD int at(int j) const { return (ids >> (4 * j)) & 15; }
};

/// What the CTA's phases read: the tables of one grid and the slots' memory.
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
  WWB_PD float* s(int k, int off) const { return w + off + k * L->ws; }
  WWB_PD float* gs(int k, int off) const { return gw + off + static_cast<size_t>(k) * L->total_g; }
  WWB_PD float* tr(int k) const { return t + k * L->tslot; }
  WWB_PD unsigned char* llws(int k) const {
    return reinterpret_cast<unsigned char*>(w + L->llws + k * L->ws);
  }
  WWB_PD int row(int i) const {
#if defined(__CUDA_ARCH__)
    return static_cast<int>(__umulhi(static_cast<unsigned>(i), L->nth_magic));
#else
    return i / L->nth;
#endif
  }
};

/// f(slot, i) for every bin i < n of the listed slots: a warp takes kLanes consecutive bins of
/// one slot, so what depends on the slot only is uniform in the warp.
template <class F>
WWB_PD void each_bin(const Grp& c, const SlotList& l, int n, F f) {
  const int nch = (n + Grp::kLanes - 1) / Grp::kLanes, all = l.n * nch;
  for (int e = c.warp(); e < all; e += c.nwarp()) {
    const int j = (e >= nch) + (e >= 2 * nch) + (e >= 3 * nch);
    const int i = (e - j * nch) * Grp::kLanes + c.lane();
    if (i < n) f(l.at(j), i);
  }
}
/// f(slot, r) for r < n of the listed slots, one pair per thread.
template <class F>
WWB_PD void each_row(const Grp& c, const SlotList& l, int n, F f) {
  for (int e = c.tid; e < l.n * n; e += c.nthr) {
    const int j = (e >= n) + (e >= 2 * n) + (e >= 3 * n);
    f(l.at(j), e - j * n);
  }
}
static_assert(kSlots <= 4, "each_bin and each_row count three slot boundaries");
/// f(slot) on warp r: lane k runs the k-th listed slot's chain.
template <class F>
WWB_PD void each_chain(const Grp& c, int r, const SlotList& l, F f) {
  if (c.role(r))
    for (int j = c.lane(); j < l.n; j += Grp::kLanes) f(l.at(j));
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
  for (int j = 0; j < nth; ++j) v = v + r[j];
  return v;
}

WWB_PD float expf_i(float x) { return dm::expf_t<WWB_EXPF_FUSE>(x); }
WWB_PD float powf_i(float x, float y) { return dm::powf_t<WWB_POWF_FUSE>(x, y); }
WWB_PD float logf_i(float x) { return dm::logf_t<WWB_LOGF_FUSE>(x); }
/// Sine and cosine without a call: its results would pass through memory.
WWB_PD void sincosf_i(float x, float* s, float* c) { dm::sincosf_t<WWB_SINCOSF_FUSE>(x, s, c); }

// ------------------------------------------------------------------ what the slots share
/// The powers of SIG that W3SPR4 takes and the analytic tail's terms that depend on J only
/// (:886-917 of W3SIN4): functions of the grid, formed once per CTA.
WWB_PD void srce_common(const Grp& c, const SrceGroup& x) {
  const SrceLayout& L = *x.L;
  const st4::Params& q = *x.q;
  const Fields& f = *x.f;
  for (int ik = c.tid; ik < L.nk; ik += c.nthr) {
    x.w[L.pwsig + ik] = dm::powf(f.sig[ik + 1], 2.0f * q.wwnmeanptail);
    x.w[L.pwdir + ik] = dm::powf(f.sig[ik + 1], q.ssdsc[11]);
  }
  if (q.sintailpar[0] < 0.5f) {
    float* const t = x.w + L.tail;
    const float signk = f.sig[L.nk];
    const float zinf = dm::logf(signk * signk / kGrav);
    const float dely = (kLogTpiOver005 - zinf) / static_cast<float>(kJtot);
    for (int j = c.tid; j < kJtot; j += c.nthr) {
      const float y = dm::expf(zinf + static_cast<float>(j) * dely);
      const float ykm = (y / kKm);
      const float ykm2 = ykm * ykm;
      const float tensk = 1.0f + ykm2;
      const float cm = sqrt_f(kGrav * tensk / y);
      t[j] = cm;
      t[kJtot + j] = 0.5f * (3.0f * ykm2 + 1.0f) * sqrt_f(kGrav / (y * tensk));
      t[4 * kJtot + j] = cm * cm;
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
WWB_PD void srce_begin(const Grp& c, const SrceGroup& x, const SlotList& l) {
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
    for (; ik < L.nk; ++ik)
      if (wn[ik] * depth > 6.0f) break;
    x.sh[k].nscut = ik == 0 ? -1 : ik * L.nth;
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
  });
  c.sync();
}

// ------------------------------------------------------------------------------------ W3SPR4
/// W3SPR4 (w3src4md.F90:142-384) of the listed slots, first phase: the per-IK direction sums and
/// the terms of the moments (:245-300); the arrays T0 .. T5 and SIGFAC stay in the slot's transient
/// region from `off` on. The libmvec powers of :316 and :317 use scalar powf in every lane; the
/// powers are functions of the grid or of the point's WN and are kept (x.w pwsig, pwdir, pwwn).
WWB_PD void spr4_sums(const Grp& c, const SrceGroup& x, const SlotList& l, int off) {
  const SrceLayout& L = *x.L;
  const Fields& f = *x.f;
  const int nk = L.nk, nth = L.nth;
  each_row(c, l, nk, [&](int k, int ik) {
    const float* const a = x.s(k, L.spec) + ik * nth;
    const unsigned char* const lw = x.llws(k) + ik * nth;
    float ebk = 0.0f, eb2k = 0.0f;
    if ((nth & 3) == 0) {
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
WWB_PD void spr4_chains(const Grp& c, const SrceGroup& x, const SlotList& l, int off) {
  const SrceLayout& L = *x.L;
  const st4::Params& p = *x.q;
  const Fields& f = *x.f;
  const int nk = L.nk, nth = L.nth;
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
  for (int comp = 0; comp < 2; ++comp) {
    each_chain(c, 1 + comp, l, [&](int k) {
      const float* const a = x.s(k, L.spec);
      const float* const sf = x.tr(k) + off + 6 * nk;
      const float* const e = comp ? f.esin : f.ecos;
      float v = 0.0f;
      for (int ik = 0; ik < nk; ++ik) {
        const float sfk = sf[ik];
        const float* const ar = a + ik * nth;
        const float* const er = e + ik * nth;
WWB_UNROLL(12)
        for (int i = 0; i < nth; ++i) v = v + ar[i] * er[i] * sfk;
      }
      x.sh[k].chains[comp] = v;
    });
  }
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
/// DSTAB and LLWS of one bin (:739-783).
WWB_PD float scan_bin(const st4::Params& p, const SrceSh& s, const ScanK& q, float ustar,
                      float ustp, float coswind, int* lw) {
  float dst;
  if (coswind > 0.01f) {
    const float xx = coswind * q.ucn;
    const float zarg = kKappa / xx;
    const float zlog = q.zcn + zarg;
    int l;
    if (zlog < 0.0f) {
      const float zlog2 = zlog * zlog;
      dst = q.cnst * expf_i(zlog) * (zlog2 * zlog2) * q.ucn * q.ucn * powf_i(coswind, p.ssinthp);
      l = 1;
    } else {
      dst = 0.0f;
      l = 0;
    }
    if (28.0f * q.cm * ustar * coswind >= 1.0f) l = 1;
    *lw = l;
  } else {
    dst = 0.0f;
    *lw = 0;
  }
  if ((p.sswellf[0] != 0.0f && dst < 1E-7f * q.sig2is) || p.sswellf[2] > 0.0f) {
    const float dvisc = q.swv;
    const float dturb = q.swt * (s.fw * s.uorb + (s.fu + s.fud * coswind) * ustp);
    dst = dst + s.pturb * dturb + s.pvisc * dvisc;
  }
  return dst;
}

/// Offsets of W3SIN4's NK arrays in a slot's transient region (after the R + R/4 floats of the
/// stress terms and their signs).
struct Sin4At {
  int zcn, cm, const2, cnst, swv, swt, tu, ta, end;
};
WWB_PD Sin4At sin4_at(const SrceLayout& L) {
  const int R = (L.nspec + 3) & ~3, K = (L.nk + 3) & ~3;
  const int o = R + ((((R + 3) / 4) + 3) & ~3);
  return Sin4At{o, o + K, o + 2 * K, o + 3 * K, o + 4 * K, o + 5 * K, o + 6 * K, o + 7 * K, o + 8 * K};
}

WWB_PD ScanK scan_k(const SrceGroup& x, const Sin4At& at, int k, int ik, float ustp) {
  const float* const t = x.tr(k) + ik;
  ScanK q;
  q.cm = t[at.cm];
  q.ucn = ustp * q.cm + x.q->zzalp;
  q.const2 = t[at.const2];
  q.cnst = t[at.cnst];
  q.zcn = t[at.zcn];
  q.swv = t[at.swv];
  q.swt = t[at.swt];
  q.sig2is = x.f->sig2[ik * x.L->nth];
  return q;
}

/// Lanes that share one point's stress scan: 36 directions in three rounds, 24 in two; two points
/// to a warp.
#if defined(__CUDA_ARCH__)
constexpr int kScanLanes = 12;
#else
constexpr int kScanLanes = 1;
#endif

/// The stress scan over IK (:696-797) for slots whose running stress feeds the next frequency
/// (TTAUWSHELTER /= 0) or that the parallel form leaves to it. A team of kScanLanes lanes takes one
/// point: every lane forms the frequency's scalars, the directions are split, and the four ordered
/// sums (x and y, by the sign of DSTAB) are one lane each.
WWB_PD void scan_serial(const Grp& c, const SrceGroup& x, const SlotList& l, const Sin4At& at) {
  const SrceLayout& L = *x.L;
  const st4::Params& p = *x.q;
  const Fields& f = *x.f;
  const int nk = L.nk, nth = L.nth, T4 = (nth + 3) & ~3;
  constexpr int kPerWarp = Grp::kLanes / kScanLanes;
  const int team = c.lane() / kScanLanes, sub = c.lane() - team * kScanLanes;
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
    const float ustar = s.r.ustar, shelter = fabs_f(p.ttauwshelter);
    float ust = ustar, taux = 0.0f, tauy = 0.0f, cosu = 0.0f, sinu = 0.0f, ustp = 0.0f;
    const int first = p.stab3 ? 1 : 3, last = p.stab3 ? 2 : 3;
    for (int istab = first; istab <= last; ++istab) {
      if (istab == 1) ust = ustar * (1.0f - s.ustarsigma);
      if (istab == 2) ust = ustar * (1.0f + s.ustarsigma);
      taux = (ust * ust) * s.cosw;
      tauy = (ust * ust) * s.sinw;
      if (on)
        for (int q = sub; q < 4; q += kScanLanes) s.sums[q] = 0.0f;
      c.syncwarp();
      for (int ik = 0; ik < nk; ++ik) {
        if (on) {
          const float taupx = taux - shelter * s.sums[0];
          const float taupy = tauy - shelter * s.sums[1];
          ustp = min_r(powf_i((taupx * taupx + taupy * taupy), 0.25f), max_r(ust, 0.3f));
          const float usdirp = dm::atan2f(taupy, taupx);
          sincosf_i(usdirp, &sinu, &cosu);
          const ScanK q = scan_k(x, at, k, ik, ustp);
          for (int ith = sub; ith < nth; ith += kScanLanes) {
            const int i = ik * nth + ith;
            const float ecos = f.ecos[i], esin = f.esin[i];
            const float coswind = (ecos * cosu + esin * sinu);
            int lw;
            const float dst = scan_bin(p, s, q, ustar, ustp, coswind, &lw);
            if (istab == 2) {
              vdin[i] = 0.5f * (vdin[i] + dst);
            } else {
              vdin[i] = dst;
            }
            llws[i] = static_cast<unsigned char>(lw);
            const float temp2 = q.const2 * dst * a[i];
            bx[ith] = temp2 * ecos;
            by[ith] = temp2 * esin;
            neg[ith] = dst < 0.0f ? 1 : 0;
          }
        }
        c.syncwarp();
        if (on)
          for (int q = sub; q < 4; q += kScanLanes) {
            float v = s.sums[q];
            const float* const b = (q & 1) ? by : bx;
            const unsigned want = static_cast<unsigned>(q >> 1);
WWB_UNROLL(12)
            for (int ith = 0; ith < nth; ++ith)
              if (neg[ith] == want) v = v + b[ith];
            s.sums[q] = v;
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

WWB_PD bool finite_f(float v) { return fabs_f(v) <= 3.402823466e38f; }

/// W3SIN4 (w3src4md.F90:423-1003) of the listed slots with W3SRCE's arguments (:1100, :1239, :2007):
/// VDIN, LLWS, TAUWX/Y, TAUWAX/Y. VSIN = VDIN * SPEC is formed where it is read (the spectrum does not
/// change before that).
WWB_PD void srce_sin4(const Grp& c, const SrceGroup& x, const SlotList& l) {
  const SrceLayout& L = *x.L;
  const st4::Params& p = *x.q;
  const Fields& f = *x.f;
  const int nk = L.nk, nth = L.nth;
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
    t[at.zcn] = logf_i(kis * s.r.z0);
    t[at.swv] = -(p.sswellf[4] * s.drat * 2.0f * kis * sqrt_f(kTwoNuAir * sig2is));
    t[at.swt] = -(s.drat * p.sswellf[0] * 16.0f * (sig2is * sig2is) / kGrav);
    t[at.tu] = e * (sigk * sigk) * f.dden[ik] / cg;
    t[at.ta] = e * f.dden[ik] / cg;
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
    s.uorb = uorb;
    s.pturb = pturb;
    s.pvisc = pvisc;
    s.fw = fw;
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
  SlotList par, ser;
  for (int j = 0; j < l.n; ++j) {
    if (x.sh[l.at(j)].scan_par) par.add(l.at(j));
    else ser.add(l.at(j));
  }
  if (par.n) {
    const int R = (L.nspec + 3) & ~3;
    each_bin(c, par, L.nspec, [&](int k, int i) {
      const SrceSh& s = x.sh[k];
      const int ik = x.row(i);
      const float ustp = s.ustp;
      const ScanK q = scan_k(x, at, k, ik, ustp);
      const float coswind = (f.ecos[i] * s.cosu + f.esin[i] * s.sinu);
      int lw;
      const float dst = scan_bin(p, s, q, s.r.ustar, ustp, coswind, &lw);
      x.gs(k, L.vdin)[i] = dst;
      x.llws(k)[i] = static_cast<unsigned char>(lw);
      x.tr(k)[i] = q.const2 * dst * x.s(k, L.spec)[i];
      reinterpret_cast<unsigned char*>(x.tr(k) + R)[i] = dst < 0.0f ? 1 : 0;
    });
    c.sync();
    for (int r = 0; r < 4; ++r) {
      each_chain(c, r, par, [&](int k) {
        const float* const e = (r & 1) ? f.esin : f.ecos;
        const float* const t2 = x.tr(k);
        const unsigned char* const neg = reinterpret_cast<const unsigned char*>(t2 + R);
        const unsigned want = static_cast<unsigned>(r >> 1);
        float v = 0.0f;
        walk4(t2, L.nspec, [&](float tv, int i) {
          if (neg[i] == want) v = v + tv * e[i];
        });
        x.sh[k].sums[r] = v;
        (r < 2 ? x.sh[k].ss : x.sh[k].sn)[2][r & 1] = v;
      });
    }
    c.sync();
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
  // 3. The tail stress and the stress limit (:799-976).
  each_chain(c, 0, l, [&](int k) {
    SrceSh& s = x.sh[k];
    const float* const a = x.s(k, L.spec);
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
    float ustl, usdirpl;
    {
      const float taupx = s.taux - fabs_f(p.ttauwshelter) * xstress;
      const float taupy = s.tauy - fabs_f(p.ttauwshelter) * ystress;
      ustl = dm::powf((taupx * taupx + taupy * taupy), 0.25f);
      usdirpl = dm::atan2f(taupy, taupx);
    }
    const float ust3 = ustl, z0 = s.r.z0, ustar = s.r.ustar;
    float c0;
    {
      const float signk = f.sig[nk];
      const float s2 = signk * signk;
      const float s5 = s2 * (s2 * signk);
      c0 = p.dth * s5 / kGrav2Tpi * kTpi * signk / x.s(k, L.cg1)[nk - 1];
    }
    float temp = 0.0f;
    for (int ith = 0; ith < nth; ++ith) {
      const int i = ith + (nk - 1) * nth;
      const float coswind = (f.ecos[i] * s.cosu + f.esin[i] * s.sinu);
      const float cp = (max_r(coswind, 0.0f));
      temp = temp + a[i] * (cp * (cp * cp));
    }
    const float levtail0 = c0 * temp;
    float tauhf;
    if (p.sintailpar[0] < 0.5f) {
      const float* const tt = x.w + L.tail;
      float ustr = ust3;
      const float signk = f.sig[nk];
      const float zinf = dm::logf(signk * signk / kGrav);
      const float dely = (kLogTpiOver005 - zinf) / static_cast<float>(kJtot);
      float taur = ust3 * ust3;
      float tau1 = 0.0f;
      const float const1 = s.const1, gz0 = kGrav * z0;
      for (int j = 1; j <= kJtot; ++j) {
        const float w = (j == 1 || j == kJtot) ? 0.5f : 1.0f;
        const float cm = tt[j - 1];
        const float cgtail = tt[kJtot + j - 1];
        const float gz = gz0 / tt[4 * kJtot + j - 1];
        const float zx = ustr / cm + p.zzalp;
        const float zarg = min_r(kKappa / zx, 20.0f);
        const float zmu = min_r(gz * expf_i(zarg), 1.0f);
        const float zlog = min_r(logf_i(zmu), 0.0f);
        const float zlog2 = zlog * zlog;
        const float zbeta = const1 * zmu * (zlog2 * zlog2);
        float levtail;
        if (p.sintailpar[2] > 0.0f) {
          float alpham;
          if (ustr < cm) {
            alpham = max_r(0.0f, 0.01f * (1.0f + dm::logf(ustr / cm)));
          } else {
            alpham = 0.01f * (1.0f + 3.0f * dm::logf(ustr / cm));
          }
          const float fm = tt[2 * kJtot + j - 1];
          const float alphat = alpham * tt[5 * kJtot + j - 1] * fm;
          const float th = tt[3 * kJtot + j - 1];
          levtail = levtail0 * 0.5f * (1.0f - th) + p.sintailpar[2] * 0.5f * (1.0f + th) * alphat;
        } else {
          levtail = levtail0;
        }
        tau1 = tau1 + w * zbeta * (ustr * ustr) * levtail * dely * cgtail / cm;
        taur = taur - w * p.sintailpar[1] * (ustr * ustr) * zbeta * levtail * dely * cgtail / cm;
        ustr = sqrt_f(max_r(taur, 0.0f));
      }
      tauhf = tau1;
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
      tauhf = levtail0 * (ust3 * ust3) * tau1;
    }
    float cp, sp;
    dm::sincosf(usdirpl, &sp, &cp);
    float twx = xstress + tauhf * cp;
    float twy = ystress + tauhf * sp;
    const float tauw = sqrt_f(twx * twx + twy * twy);
    const float ust2b = max_r(ustar, kEps2);
    const float ust2 = ust2b * ust2b;
    const float tauwb = min_r(tauw, max_r(ust2 - kEps1, kEps2Sq));
    if (tauwb < tauw) {
      twx = twx * tauwb / tauw;
      twy = twy * tauwb / tauw;
    }
    s.tauwx = twx;
    s.tauwy = twy;
  });
  c.sync();
}

// ------------------------------------------------------------------------- the DIA (W3SNL1)
/// The step's DIA (:1259-1263) with KDMEAN = WNMEAN * DEPTH for the listed slots (the arithmetic of
/// snl1_rowshift_kernel): VSNL and VDNL. UE, SA1, SA2 of as many slots as fit sit in the transient
/// region; DA1P, DA1M, DA2P, DA2M and DA1C + DA2C in the slot's global scratch (DA1C and DA2C are read
/// back only at their own bin, so their sum is kept, the same two roundings).
WWB_PD void srce_dia(const Grp& c, const SrceGroup& x, const SlotList& all) {
  const SrceLayout& L = *x.L;
  const Snl1Dev& p = *x.n;
  const int nth = p.nth, nfr = p.nfr, nfrhgh = p.nfrhgh, nfrchg = p.nfrchg;
  const int nspec = p.nspec, nspecx = p.nspecx, nk = p.nk;
  const int A4 = (L.alen + 3) & ~3, U4 = ((nfrhgh + 1) * nth + 3) & ~3;
  const int per = srce_trans_floats(L, x.ns) / L.dia;
  const float dal1 = p.dal1, dal2 = p.dal2, dal3 = p.dal3;
  for (int j0 = 0; j0 < all.n; j0 += per) {
    SlotList l;
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
    each_bin(c, l, nspec, [&](int k, int i) {
      float* const ue = ue_of(k);
      ue[i + nth] = x.s(k, L.spec)[i] / ue[U4 + 2 * A4 + x.row(i)];
    });
    c.sync();
    each_row(c, l, nth, [&](int k, int col) {
      float* const ue = ue_of(k);
      float t = ue[nfr * nth + col];
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
    each_bin(c, l, nspecx, [&](int k, int isp) {
      float* const ue = ue_of(k);
      float* const sa1 = ue + U4;
      float* const sa2 = sa1 + A4;
      const int ifr0 = x.row(isp), ith = isp - ifr0 * nth;
      int cc[8];
      for (int n = 0; n < 8; ++n) {
        const int v = ith + p.shift[n];
        cc[n] = v < 0 ? v + nth : (v >= nth ? v - nth : v);
      }
      const int r1 = p.ifrow[0 * nfrchg + ifr0] * nth;
      const int r2 = p.ifrow[1 * nfrchg + ifr0] * nth;
      const int r3 = p.ifrow[2 * nfrchg + ifr0] * nth;
      const int r4 = p.ifrow[3 * nfrchg + ifr0] * nth;
      const float e00 = ue[isp + nth];
      const float ep1 = p.awg[0] * ue[r2 + cc[1]] + p.awg[1] * ue[r2 + cc[0]] +
                        p.awg[2] * ue[r1 + cc[1]] + p.awg[3] * ue[r1 + cc[0]];
      const float em1 = p.awg[4] * ue[r4 + cc[7]] + p.awg[5] * ue[r4 + cc[6]] +
                        p.awg[6] * ue[r3 + cc[7]] + p.awg[7] * ue[r3 + cc[6]];
      const float ep2 = p.awg[0] * ue[r2 + cc[5]] + p.awg[1] * ue[r2 + cc[4]] +
                        p.awg[2] * ue[r1 + cc[5]] + p.awg[3] * ue[r1 + cc[4]];
      const float em2 = p.awg[4] * ue[r4 + cc[3]] + p.awg[5] * ue[r4 + cc[2]] +
                        p.awg[6] * ue[r3 + cc[3]] + p.awg[7] * ue[r3 + cc[2]];
      const float ca = x.sh[k].cons * p.af11_row[ifr0];
      const float factor = ca * e00;
      const float sa1a = e00 * (ep1 * dal1 + em1 * dal2);
      const float sa1b = sa1a - ep1 * em1 * dal3;
      const float sa2a = e00 * (ep2 * dal1 + em2 * dal2);
      const float sa2b = sa2a - ep2 * em2 * dal3;
      const int o = isp + nth;
      sa1[o] = factor * sa1b;
      sa2[o] = factor * sa2b;
      float* const da = x.gs(k, L.da);
      if (isp < nspec) da[4 * A4 + isp] = ca * (sa1a + sa1b) + ca * (sa2a + sa2b);
      da[o] = factor * (dal1 * e00 - dal3 * em1);
      da[A4 + o] = factor * (dal2 * e00 - dal3 * ep1);
      da[2 * A4 + o] = factor * (dal1 * e00 - dal3 * em2);
      da[3 * A4 + o] = factor * (dal2 * e00 - dal3 * ep2);
    });
    c.sync();
    each_bin(c, l, nspec, [&](int k, int isp) {
      const float* const ue = ue_of(k);
      const float* const sa1 = ue + U4;
      const float* const sa2 = sa1 + A4;
      const float* const da1p = x.gs(k, L.da);
      const float* const da1m = da1p + A4;
      const float* const da2p = da1m + A4;
      const float* const da2m = da2p + A4;
      const int ifr0 = x.row(isp), ith = isp - ifr0 * nth;
      int cc[8];
      for (int n = 0; n < 8; ++n) {
        const int v = ith + p.shift[n];
        cc[n] = v < 0 ? v + nth : (v >= nth ? v - nth : v);
      }
      const int r5 = p.ifrow[4 * nfrchg + ifr0] * nth;
      const int r6 = p.ifrow[5 * nfrchg + ifr0] * nth;
      const int r7 = p.ifrow[6 * nfrchg + ifr0] * nth;
      const int r8 = p.ifrow[7 * nfrchg + ifr0] * nth;
      const int o = isp + nth;
      x.gs(k, L.vsnl)[isp] = ue[U4 + 2 * A4 + ifr0] * (-2.0f * (sa1[o] + sa2[o]) +
                             p.awg[0] * (sa1[r6 + cc[5]] + sa2[r6 + cc[1]]) +
                             p.awg[1] * (sa1[r6 + cc[4]] + sa2[r6 + cc[0]]) +
                             p.awg[2] * (sa1[r5 + cc[5]] + sa2[r5 + cc[1]]) +
                             p.awg[3] * (sa1[r5 + cc[4]] + sa2[r5 + cc[0]]) +
                             p.awg[4] * (sa1[r8 + cc[3]] + sa2[r8 + cc[7]]) +
                             p.awg[5] * (sa1[r8 + cc[2]] + sa2[r8 + cc[6]]) +
                             p.awg[6] * (sa1[r7 + cc[3]] + sa2[r7 + cc[7]]) +
                             p.awg[7] * (sa1[r7 + cc[2]] + sa2[r7 + cc[6]]));
      x.gs(k, L.vdnl)[isp] = -2.0f * da1p[4 * A4 + isp] +
                             p.swg[0] * (da1p[r6 + cc[5]] + da2p[r6 + cc[1]]) +
                             p.swg[1] * (da1p[r6 + cc[4]] + da2p[r6 + cc[0]]) +
                             p.swg[2] * (da1p[r5 + cc[5]] + da2p[r5 + cc[1]]) +
                             p.swg[3] * (da1p[r5 + cc[4]] + da2p[r5 + cc[0]]) +
                             p.swg[4] * (da1m[r8 + cc[3]] + da2m[r8 + cc[7]]) +
                             p.swg[5] * (da1m[r8 + cc[2]] + da2m[r8 + cc[6]]) +
                             p.swg[6] * (da1m[r7 + cc[3]] + da2m[r7 + cc[7]]) +
                             p.swg[7] * (da1m[r7 + cc[2]] + da2m[r7 + cc[6]]);
    });
    c.sync();
  }
}

// ------------------------------------------------------------------------------------ W3SDS4
/// The cumulative term's sums over B-wide blocks of one IK2 row for up to kSlots points:
/// v[j] += sum over the row of CUMULW * BRLAMBDA in order, for the slots of `mask`.
template <int B>
WWB_PD void cumul_row(const float* cw, size_t step, const float* const* brl, int nth,
                      unsigned mask, float* v) {
  for (int j0 = 0; j0 < nth; j0 += B) {
    float q[B];
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
    for (int b = 0; b < B; ++b) q[b] = cw[static_cast<size_t>(j0 + b) * step];
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
    for (int j = 0; j < kSlots; ++j) {
      if (!(mask >> j & 1)) continue;
      float a = v[j];
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
      for (int b = 0; b < B; b += (B >= 4 ? 4 : 1)) {
        if (B >= 4) {
          const F4 r = ld4(brl[j] + j0 + b);
          a = a + q[b] * r.a;
          a = a + q[b + (B >= 4 ? 1 : 0)] * r.b;
          a = a + q[b + (B >= 4 ? 2 : 0)] * r.c;
          a = a + q[b + (B >= 4 ? 3 : 0)] * r.d;
        } else {
          a = a + q[b] * brl[j][j0 + b];
        }
      }
      v[j] = a;
    }
  }
}

/// W3SDS4 (w3src4md.F90:2043-2659) of the listed slots: VSDS, VDDS, WHITECAP. BRLAMBDA stays in the
/// slot's transient region (BTH before it, in place), the NK arrays behind it. The libmvec loops
/// (:2315, :2500, :2509) use scalar powf/expf in every lane.
WWB_PD void srce_sds4(const Grp& c, const SrceGroup& x, const SlotList& l) {
  const SrceLayout& L = *x.L;
  const st4::Params& p = *x.q;
  const Fields& f = *x.f;
  const int nk = L.nk, nth = L.nth, nspec = L.nspec;
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
      each_bin(c, l, nspec, [&](int k, int i) {
        const int ik0 = x.row(i), ith0 = i - ik0 * nth;
        float v = zero;
        if (ik0 + 1 >= ik1) {
          const float* const a = x.s(k, L.spec) + ik0 * nth - 1;
          const float* const sw = f.satw_t + ith0;
          const int* const si = f.sati_t + ith0;
WWB_UNROLL(6)
          for (int j = 0; j < rows; ++j) v = v + sw[j * f.sat_ld] * a[si[j * f.sat_ld]];
          const float kx = x.s(k, L.wn1)[ik0];
          const float facsat = (f.sig[ik0 + 1] * ((kx * kx) * kx)) * dth;
          v = v * facsat;
        }
        brl_of(k)[i] = v;
      });
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
          for (; i < is0 + nth; ++i) {
            if (bth[i] >= lim) {
              lim = bth[i];
              ++i;
              found = true;
              break;
            }
          }
          if (!found) lim = dm::asfloat(0x7fc00000u);
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
    each_bin(c, l, nspec, [&](int k, int i) {
      const int ik0 = x.row(i);
      const bool in = ik0 + 1 >= ik1;
      float bth = zero, dd = zero;
      if (in) {
        bth = p.ssdsdth >= 180.0f ? nka(k, kBth0)[ik0] : brl_of(k)[i];
        dd = nka(k, kA2)[ik0] +
             nka(k, kA3)[ik0] * powf_i(max_r(bth - nka(k, kA1)[ik0], zero), p.ssdsp);
      }
      const float m = max_r(sqrt_f(bth) - epsr, zero);
      float pbi = m * m;
      pbi = pbi * 28.16f;
      brl_of(k)[i] = pbi / kTwoPiSq;
      x.gs(k, L.vdds)[i] = dd;
      x.gs(k, L.vsds)[i] = dd * x.s(k, L.spec)[i];
    });
    c.sync();
  } else if (sdscase == 2) {
    // 2.b Filipot et al. (:2338-2477). E1 = kB1, DK = kB2, the serial part's arrays behind.
    each_row(c, l, nk, [&](int k, int ik0) {
      const int ik = ik0 + 1;
      float e = zero, dk = zero;
      if (ik >= ik1) {
        const float* const a = x.s(k, L.spec) + ik0 * nth;
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
      for (int i = 0; i < nk; ++i) hs[i] = efdf[i] = kbar[i] = zero;
      for (int ikl = 1; ikl <= nk; ++ikl) {
        iksup[ikl - 1] = f.iktab[(ikl - 1) + (id - 1) * f.iktab_ld];
        if (iksup[ikl - 1] <= nk) {
          float v = zero;
          for (int i = ikl; i <= iksup[ikl - 1] - 1; ++i) v = v + e1[i - 1] * dk[i - 1];
          efdf[ikl - 1] = v;
          if (efdf[ikl - 1] != zero) {
            float w = zero;
            for (int i = ikl; i <= iksup[ikl - 1] - 1; ++i) w = w + (kk[i - 1] * e1[i - 1]) * dk[i - 1];
            kbar[ikl - 1] = w / efdf[ikl - 1];
          } else {
            kbar[ikl - 1] = zero;
          }
          hs[ikl - 1] = 4.0f * sqrt_f(efdf[ikl - 1]);
          nkl = nkl + 1;
        }
      }
      for (int i = 0; i < nk; ++i) dck[i] = qb[i] = zero;
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
      for (int i = 0; i < nk; ++i) {
        s1[i] = s2[i] = zero;
        ntimes[i] = 0;
      }
      for (int ikl = 1; ikl <= nkl; ++ikl) {
        if (efdf[ikl - 1] > zero) {
          for (int i = ikl; i <= iksup[ikl - 1]; ++i)
            s1[i - 1] = s1[i - 1] + (dck[ikl - 1] * e1[i - 1]) / efdf[ikl - 1];
          for (int i = ikl; i <= iksup[ikl - 1]; ++i)
            s2[i - 1] = s2[i - 1] + (qb[ikl - 1] * e1[i - 1]) / efdf[ikl - 1];
          for (int i = ikl; i <= iksup[ikl - 1]; ++i) ntimes[i - 1] = ntimes[i - 1] + 1;
        }
      }
      for (int i = 0; i < nk; ++i) {
        if (ntimes[i] > 0) {
          s1[i] = s1[i] / static_cast<float>(ntimes[i]);
          s2[i] = s2[i] / static_cast<float>(ntimes[i]);
        } else {
          s1[i] = s2[i] = zero;
        }
      }
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
      float b = (((c9 * expf_i(-(p.ssdsbr / bthk))) * nka(k, kB4)[ik0]) / c13p1) * lmod;
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
        for (int i = 0; i < nth; ++i) w = w + (b[i] * (-ssdsc[1])) * pw;
        c5 = ((((cc * cc) * cc) * w) * p.aairgb / kGrav) * f.dden[ik0] / (f.sig[ik] * cg);
      }
      nka(k, kCoef4)[ik0] = c4;
      nka(k, kCoef5)[ik0] = c5;
    });
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
    // Each thread takes a bin of every slot: CUMULW's row is read once for all of them, BRLAMBDA is a
    // broadcast. The bins of the highest frequencies have the longest sums and come first.
    const float* brl[kSlots];
    for (int j = 0; j < kSlots; ++j) brl[j] = brl_of(l.at(j < l.n ? j : 0));
    const int nch = (nspec + Grp::kLanes - 1) / Grp::kLanes;
    for (int e = nch - 1 - c.warp(); e >= 0; e -= c.nwarp()) {
      const int i = e * Grp::kLanes + c.lane();
      if (i >= nspec) continue;
      const int ik0 = x.row(i), ik = ik0 + 1, ith0 = i - ik0 * nth;
      if (ik < ik1) continue;
      float ren[kSlots] = {0.0f, 0.0f, 0.0f, 0.0f};
      if (ssdsc[2] < zero && ik > dikcumul) {
        for (int ik2 = ik1; ik2 <= ik - dikcumul; ++ik2) {
          unsigned mask = 0;
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
          for (int j = 0; j < kSlots; ++j)
            if (j < l.n && brl[j][R + kBth0 * K + ik2 - 1] > p.ssdsbr) mask |= 1u << j;
          if (mask == 0) continue;
          const int is2 = (ik2 - 1) * nth;
          const float* row[kSlots];
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
          for (int j = 0; j < kSlots; ++j) row[j] = brl[j] + is2;
          float v[kSlots] = {0.0f, 0.0f, 0.0f, 0.0f};
          // CUMULW(IS2+J, IS) as a function of IK2, IK and J - ITH where the table is one (f.cumt), else
          // the transposed table: consecutive IS are consecutive in both.
          const float* cw;
          size_t step;
          if (f.cumt != nullptr) {
            const int ld = 2 * nth - 1;
            cw = f.cumt + (static_cast<size_t>(ik2 - 1) * nk + ik0) * ld + (nth - 1 - ith0);
            step = 1;
          } else {
            cw = f.cumulw + static_cast<size_t>(is2) * f.cumulw_ld + i;
            step = f.cumulw_ld;
          }
          if (nth % 12 == 0) cumul_row<12>(cw, step, row, nth, mask, v);
          else if (nth % 4 == 0) cumul_row<4>(cw, step, row, nth, mask, v);
          else cumul_row<1>(cw, step, row, nth, mask, v);
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
          for (int j = 0; j < kSlots; ++j)
            if (mask >> j & 1) ren[j] = ren[j] + v[j];
        }
      }
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
      for (int j = 0; j < kSlots; ++j) {
        if (j >= l.n) continue;
        const int k = l.at(j);
        const SrceSh& s = x.sh[k];
        const float kx = x.s(k, L.wn1)[ik0];
        const float facturb2 = -(((f.sig[ik] * 2.0f) * kx) * s.facturb);
        const float dvisc = -(((ssdsc[20] * 4.0f) * kx) * kx);
        const float renewalfreq = ssdsc[2] > zero ? nka(k, kRen)[ik0] : ren[j];
        const float coswind = f.ecos[ith0] * s.cosus + f.esin[ith0] * s.sinus;
        const float dturb = facturb2 * max_r(coswind, zero);
        const float diag2 = (ssdsc[2] * renewalfreq + dturb) + dvisc;
        float* const vdds = x.gs(k, L.vdds) + i;
        float* const vsds = x.gs(k, L.vsds) + i;
        *vdds = *vdds + diag2;
        *vsds = *vsds + x.s(k, L.spec)[i] * diag2;
      }
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
        for (int ik = ik1; ik <= ikc; ++ik) {
          wc0 = wc0 + coef4[ik - 1] * (one - wc0);
          wc3 = wc3 + coef5[ik - 1];
        }
      }
      if (s.in.flogrd58) {
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
/// A step up to the update (:1210-1847) of the listed slots: the step count, W3SLN1, the DIA, W3SDS4,
/// W3SDB1, W3SBT1, the time step, the new spectrum and the terms of the closing sums.
WWB_PD void srce_advance(const Grp& c, const SrceGroup& x, const SlotList& l) {
  const srce::Params& p = *x.p;
  const SrceLayout& L = *x.L;
  const int nk = L.nk, nth = L.nth, nspec = L.nspec;
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
    const int nch = (nspec + Grp::kLanes - 1) / Grp::kLanes, all = l.n * nch;
    for (int e = c.warp(); e < all; e += c.nwarp()) {
      const int j = (e >= nch) + (e >= 2 * nch) + (e >= 3 * nch);
      const int k = l.at(j), i = (e - j * nch) * Grp::kLanes + c.lane();
      SrceSh& s = x.sh[k];
      float v = dm::asfloat(0x7f800000u);
      if (i < s.nspech) {
        const int ik = x.row(i);
        const float spec = x.s(k, L.spec)[i];
        const int nscut = s.nscut;
        float vdin = x.gs(k, L.vdin)[i];
        float vsin = vdin * spec;
        float vsnl = x.gs(k, L.vsnl)[i], vdnl = x.gs(k, L.vdnl)[i];
        float vsds = x.gs(k, L.vsds)[i], vdds = x.gs(k, L.vdds)[i];
        float vsln = p.ln1 ? x.s(k, L.wnf)[ik] * x.s(k, L.dirf)[i - ik * nth] : 0.0f;
        float vdbt = 0.0f, vsbt = 0.0f;
        if (nscut >= 0) {
          vdbt = i < nscut ? x.s(k, L.cbeta)[x.g->mapwn[i] - 1] : 0.0f;
          vsbt = vdbt * spec;
        }
        if (s.in.inflags24) {
          vsnl = s.icescalenl * vsnl;
          vdnl = s.icescalenl * vdnl;
          vsln = s.icescaleln * vsln;
          vsin = s.icescalein * vsin;
          vdin = s.icescalein * vdin;
          vsds = s.icescaleds * vsds;
          vdds = s.icescaleds * vdds;
        }
        const float vs = (((vsln + vsin) + vsnl) + vsds) + vsbt;
        const float vd = ((vdin + vdnl) + vdds) + vdbt;
        x.gs(k, L.vsds)[i] = vs;
        x.gs(k, L.vdds)[i] = vd;
        const float damax =
            mn(mx(p.xrel * x.gs(k, L.specinit)[i], s.afilt), x.s(k, L.dam)[ik]);
        const float afac = 1.0f / mx(fabs_f(vs / damax), 1.E-10f);
        v = afac / mx(mn(vd, 0.0f) * afac + 1.0f, 1.E-10f);
      }
      // The limits are never negative and never NaN (mx and mn take their second operand for
      // one), so their order is that of their bits.
#if defined(__CUDA_ARCH__)
      const unsigned m = __reduce_min_sync(0xffffffffu, dm::asuint(v));
      if (c.lane() == 0) atomicMin(&s.vmin, m);
#else
      if (dm::asuint(v) < s.vmin) s.vmin = dm::asuint(v);
#endif
    }
  }
  c.sync();
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
  each_bin(c, l, nspec, [&](int k, int i) {
    const SrceSh& s = x.sh[k];
    const int ik = x.row(i);
    const float dt = s.dt, hdt = dt;
    float* const sp = x.s(k, L.spec) + i;
    const float spec = *sp;
    const bool low = i < s.nspech;
    float vdin = x.gs(k, L.vdin)[i];
    float vsin = vdin * spec;
    if (s.in.inflags24 && low) {
      vsin = s.icescalein * vsin;
      vdin = s.icescalein * vdin;
    }
    float vsdb;
    if (s.early) {
      vsdb = x.gs(k, L.vsdb)[i];
    } else {
      vsdb = s.vddb * spec;
      x.gs(k, L.vsdb)[i] = vsdb;
    }
    const int nscut = s.nscut;
    float vdbt = 0.0f, vsbt = 0.0f;
    if (nscut >= 0) {
      vdbt = i < nscut ? x.s(k, L.cbeta)[x.g->mapwn[i] - 1] : 0.0f;
      vsbt = vdbt * spec;
    }
    if (low) {
      const float vs = x.gs(k, L.vsds)[i], vd = x.gs(k, L.vdds)[i];
      const float einc1 = (dt * vs) / mx(1.0f - hdt * vd, 1.0f);
      float v;
      if (s.shave) {
        const float einc2 = copysignf(mn(fabs_f(einc1), x.s(k, L.dam)[ik]), einc1);
        v = mx(spec + einc2, 0.0f);
      } else {
        v = mx(spec + einc1, 0.0f);
      }
      const float e2 = (dt * vsdb) / mx(1.0f - hdt * s.vddb, 1.0f);
      *sp = mx(v + e2, 0.0f);
    }
    const float factor = x.g->dden[ik] / x.s(k, L.cg1)[ik];
    float* const t = x.tr(k);
    t[i] = ((vsin * dt) * factor) / mx(1.0f - vdin * dt, 1.0f);
    t[R + i] = ((vsbt * dt) * factor) / mx(1.0f - vdbt * dt, 1.0f);
    reinterpret_cast<unsigned char*>(t + 2 * R)[i] = vsin > 0.0f ? 1 : 0;
  });
  c.sync();
}

/// The closing sums' chains (:1815-1847), roles 4-6.
WWB_PD void srce_sums(const Grp& c, const SrceGroup& x, const SlotList& l) {
  const SrceLayout& L = *x.L;
  const int R = (L.nspec + 3) & ~3;
  each_chain(c, 4, l, [&](int k) {
    float v = x.sh[k].phiaw;
    walk4(x.tr(k), L.nspec, [&](float t, int) { v = t + v; });
    x.sh[k].phiaw = v;
  });
  each_chain(c, 5, l, [&](int k) {
    float v = x.sh[k].phibbl;
    walk4(x.tr(k) + R, L.nspec, [&](float t, int) { v = v - t; });
    x.sh[k].phibbl = v;
  });
  each_chain(c, 6, l, [&](int k) {
    // A bin without wind input adds -0, which changes nothing.
    const float* const sp = x.s(k, L.spec);
    const unsigned char* const wind = reinterpret_cast<const unsigned char*>(x.tr(k) + 2 * R);
    float v = 0.0f;
    for (int ik = 0; ik < L.nk; ++ik) {
      const float factor = x.g->dden[ik] / x.s(k, L.cg1)[ik];
WWB_UNROLL(12)
      for (int i = ik * L.nth; i < (ik + 1) * L.nth; ++i)
        if (wind[i]) v = v + sp[i] * factor;
    }
    x.sh[k].whitecap[2] = sqrt_f(v) * 4.0f;
  });
}

/// After the step's W3SPR4 (:1880-1997): FHIGH, MLIM, SEED, the tail for running slots; SPECINIT and
/// FHIGH's first value for the slots that end their initialisation (:1122-1179).
WWB_PD void srce_shape(const Grp& c, const SrceGroup& x, const SlotList& run,
                       const SlotList& fresh2) {
  const srce::Params& p = *x.p;
  const SrceLayout& L = *x.L;
  const int nk = L.nk, nth = L.nth, nspec = L.nspec;
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
  SlotList lim;
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
    for (int ik = nkh; ik < nk; ++ik) {
      v = v * p.fachfa + 0.0f;
      sp[ik * nth] = v;
    }
  });
  c.sync();
}

/// 3. After the loop (:2050-2350), FLD2 excepted (ww_srce_init refuses it).
WWB_PD void srce_finish(const Grp& c, const SrceGroup& x, const SlotList& l) {
  const srce::Params& p = *x.p;
  const SrceLayout& L = *x.L;
  const int nk = L.nk, nth = L.nth, nspec = L.nspec;
  // Per-IK band sums: eband, a1band, b1band.
  each_row(c, l, nk, [&](int k, int ik) {
    const float* const spec = x.s(k, L.spec);
    const float* const specinit = x.gs(k, L.specinit);
    float eband = 0.0f, a1band = 0.0f, b1band = 0.0f;
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
      for (int ik = 0; ik < nk; ++ik) {
        const float factor = x.g->dden[ik] / x.s(k, L.cg1)[ik];
        const float factor2 = ((factor * kGrav) * x.s(k, L.wn1)[ik]) / x.g->sig[ik];
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
template <class Src>
WWB_PD void srce_run(const Grp& c, const SrceGroup& x, Src& src) {
  const SrceLayout& L = *x.L;
  const int R = (L.nspec + 3) & ~3;
  const int spr4_off = 2 * R + ((((R + 3) / 4) + 3) & ~3);
  const bool sin4_at_init = x.q->sintailpar[3] > 0.5f;  // :1100
  const bool spr4_twice = x.q->sintailpar[3] < 0.5f;    // :2012
  srce_common(c, x);
  for (;;) {
    SlotList fresh;
    src.load(c, x, fresh);
    if (fresh.n) srce_begin(c, x, fresh);
    SlotList all, run, fresh2, wind, done;
    for (int k = 0; k < x.ns; ++k) {
      const int st = x.sh[k].state;
      if (st == kIdle) continue;
      all.add(k);
      if (st == kRun) run.add(k);
      if (st == kFresh2) fresh2.add(k);
      if (st != kFresh1 || sin4_at_init) wind.add(k);
    }
    if (all.n == 0) break;
    if (run.n) srce_advance(c, x, run);
    // W3SPR4, what follows it, W3SIN4; for SINTAILPAR(4) < 0.5 running slots take W3SPR4 and (unless
    // they end) the next step's W3SIN4 once more. Otherwise the next step's W3SIN4 is this one: it
    // reads the same spectrum, USTAR, Z0 and wind, so it gives the same bits.
    for (int rep = 0;; ++rep) {
      const SlotList& spr = rep == 0 ? all : run;
      spr4_sums(c, x, spr, spr4_off);
      c.sync();
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
        for (int j = 0; j < run.n; ++j)
          if (x.sh[run.at(j)].done) done.add(run.at(j));
      }
      SlotList next = wind;
      if (rep == 1) {
        next = SlotList();
        for (int j = 0; j < run.n; ++j)
          if (!x.sh[run.at(j)].done) next.add(run.at(j));
        c.sync();
      }
      if (next.n) srce_sin4(c, x, next);
      if (!(rep == 0 && spr4_twice && run.n)) break;
    }
    each_chain(c, 0, all, [&](int k) {
      const int st = x.sh[k].state;
      x.sh[k].state = st == kFresh1 ? kFresh2 : kRun;
    });
    c.sync();
    if (done.n) {
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
  WWB_PD void load(const Grp&, const SrceGroup& x, SlotList& fresh) {
    if (taken) return;
    taken = true;
    x.sh[0].in = in;
    x.sh[0].state = in.it != 0 ? kFresh1 : kFresh2;
    fresh.add(0);
  }
  WWB_PD void store(const Grp&, const SrceGroup& x, const SlotList&) { x.sh[0].state = kIdle; }
};

/// W3SRCE for one point by one thread (the host build).
inline void srce_point(const Cta&, const SrceCtx& x) {
  const Grp c{0, 1};
  const SrceGroup g{x.p, x.g, x.q, x.f, x.n, x.L, x.w, x.gw, x.w + x.L->common + x.L->ws, x.sh, 1};
  OnePoint src{x.in};
  srce_run(c, g, src);
}

}  // namespace pt
}  // namespace wwb
