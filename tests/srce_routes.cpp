// tests/srce_routes.cpp -- the host build of the W3SRCE source (tests/hemu.cpp) with the tables that
// ww_st4_commit derives from the registered ones (CUMULW by direction difference, the rows of SATWEIGHTS
// that are summed, the repeated ECOS/ESIN row) switched on or off, and the branch-free libm forms beside
// the general ones. Compiled by tests/test_srce_routes.py.
#include "hemu.cpp"

#include <algorithm>
#include <cstdint>

extern "C" {

/// The derived tables on (returns a bit per table that applies) or off.
int routes_derived(int on) {
  static std::vector<float> cumt;
  cumt = st4::toeplitz_cumulw(g_grid);
  const bool fin = st4::finite_cumulw(g_grid), trig = st4::repeated_trig(g_grid);
  const int rows = st4::sat_rows(g_grid);
  g_fields.cumt = on && !cumt.empty() ? cumt.data() : nullptr;
  g_fields.cum_finite = on && fin;
  g_fields.trig_rows = on && trig;
  g_fields.nsat_eff = on ? rows : g_fields.nsat;
  return (cumt.empty() ? 0 : 1) | (fin ? 2 : 0) | (trig ? 4 : 0) | (rows < g_fields.nsat ? 8 : 0);
}

/// The bytes of the working set's layout (at most cap of them); returns their number.
int routes_layout(unsigned char* out, int cap) {
  const pt::SrceLayout L = pt::srce_layout(g_p, g_ndev);
  std::memcpy(out, &L, std::min<size_t>(cap, sizeof L));
  return static_cast<int>(sizeof L);
}

/// W3SIN4, W3SDS4 and W3SPR4 as W3SRCE's phases form them, for one point in one slot: spec (NSPEC), wn1 and
/// cg1 (NK), the point's packet pin, what W3SPR4 left (ustar, usdir, dlwmean, z0) and the stress entering
/// W3SPR4. Out: D, LLWS, tau[4] = TAUWX TAUWY TAUWNX TAUWNY; SRHS, DDIAG, BRLAMBDA, WHITECAP; W3SPR4's 12.
void routes_terms(const float* spec, const float* wn1, const float* cg1, const float* pin, float ustar,
                  float usdir, float dlwmean, float z0, float tauwx, float tauwy, const int* llws_in,
                  float* d, int* llws, float* tau, float* srhs, float* ddiag, float* brlambda,
                  float* whitecap, float* spr4) {
  const pt::SrceLayout L = pt::srce_layout(g_p, g_ndev);
  std::vector<float> w(L.total_s + 4), gw(L.total_g + 4);
  static pt::SrceSh sh;
  sh = pt::SrceSh{};
  const pt::Grp c{0, 1};
  const pt::SrceGroup<0> x{&g_sp, &g_sgrid, &g_p, &g_fields, &g_ndev, &L, w.data(), gw.data(),
                           w.data() + L.common + L.ws, &sh, 1, nullptr};
  std::memcpy(x.s(0, L.spec), spec, sizeof(float) * L.nspec);
  std::memcpy(x.s(0, L.wn1), wn1, sizeof(float) * L.nk);
  std::memcpy(x.s(0, L.cg1), cg1, sizeof(float) * L.nk);
  pt::SlotList l{};
  l.add(0);
  sh.in = pt::srce_in(1, 0, 1, 1, 900.0f, pin);
  pt::srce_common(c, x);
  pt::srce_begin(c, x, l);
  sh.r.ustar = ustar;
  sh.r.usdir = usdir;
  sh.r.dlwmean = dlwmean;
  sh.r.z0 = z0;
  pt::srce_sin4(c, x, l);
  std::memcpy(d, x.gs(0, L.vdin), sizeof(float) * L.nspec);
  for (int i = 0; i < L.nspec; ++i) llws[i] = x.llws(0)[i];
  const float t[4] = {sh.tauwx, sh.tauwy, sh.tauwax, sh.tauway};
  std::memcpy(tau, t, sizeof t);
  pt::srce_sds4(c, x, l);
  std::memcpy(srhs, x.gs(0, L.vsds), sizeof(float) * L.nspec);
  std::memcpy(ddiag, x.gs(0, L.vdds), sizeof(float) * L.nspec);
  std::memcpy(brlambda, x.tr(0), sizeof(float) * L.nspec);
  std::memcpy(whitecap, sh.whitecap, sizeof sh.whitecap);
  for (int i = 0; i < L.nspec; ++i) x.llws(0)[i] = static_cast<unsigned char>(llws_in[i]);
  sh.tauwx = tauwx;
  sh.tauwy = tauwy;
  pt::spr4_sums(c, x, l, 0);
  pt::spr4_chains(c, x, l, 0);
  sh.r.dlwmean = dm::atan2f(sh.chains[1], sh.chains[0]);
  sh.r.amax = sh.chains[2];
  std::memcpy(spr4, &sh.r, sizeof sh.r);
}

/// Mismatches over n seeded arguments of: 0 div_core (reciprocal seed an ulp off either way), 1 expf_q /
/// expf_neg, 2 logf_q, 3 powf_core / powf_mid, 4 sincosf_core, 5 atan2f_core, 6 div_by.
void routes_libm(long n, unsigned long long seed, long* bad) {
  using namespace dm;  // glibc's names are also in reach: the calls below say whose they mean
  uint64_t s = seed;
  auto next = [&] {
    s ^= s << 13;
    s ^= s >> 7;
    s ^= s << 17;
    return s;
  };
  auto diff = [](float a, float b) { return asuint(a) != asuint(b) && !(a != a && b != b); };
  for (int k = 0; k < 7; ++k) bad[k] = 0;
  for (long i = 0; i < n; ++i) {
    const uint64_t u = next(), v = next();
    const float any = asfloat(static_cast<uint32_t>(u));
    float a = asfloat((static_cast<uint32_t>(u) & 0x807fffffu) | (67u + (u >> 33) % 121u) << 23);
    float b = asfloat((static_cast<uint32_t>(v) & 0x807fffffu) | (67u + (v >> 33) % 121u) << 23);
    if (i % 4 == 0) b = asfloat((asuint(b) | 0x7fffffu) - static_cast<uint32_t>((v >> 50) % 4));
    if (i % 8 == 1) a = asfloat((asuint(a) & ~0x7fffffu) | static_cast<uint32_t>((u >> 40) % 8));
    if (div_ok(a, b))
      for (int d = -1; d <= 1; ++d) {
        float y = asfloat(asuint(1.0f / b) + d);
        y = fma_f(fma_f(-b, y, 1.0f), y, y);
        y = fma_f(fma_f(-b, y, 1.0f), y, y);
        float q = a * y;
        q = fma_f(fma_f(-b, q, a), y, q);
        bad[0] += diff(fma_f(fma_f(-b, q, a), y, q), a / b);
        if (d == 0) bad[0] += diff(div_core(a, b), a / b);
      }
    bad[1] += diff(expf_q(any), dm::expf(any));
    if (any == any) bad[1] += diff(expf_neg(-fabsf(any)), dm::expf(-fabsf(any)));
    bad[2] += diff(logf_q(any), dm::logf(any));
    if (normal_pos(any)) bad[3] += diff(powf_core(any, 0.25f), dm::powf(any, 0.25f));
    const float x = 0.0078125f + static_cast<float>(u % 10000000) * 1.9e-7f,
                y = 0.001f + static_cast<float>(v % 1000000) * 1.59e-5f;
    if (x < 2.0f && y < 16.0f) bad[3] += diff(powf_mid(x, y), dm::powf(x, y));
    const float w = i & 1 ? any : static_cast<float>(static_cast<int>(u % 2000001) - 1000000) * 3.3e-6f;
    if (abstop12(w) < abstop12(120.0f)) {
      float s1, c1, s2, c2;
      dm::sincosf(w, &s1, &c1);
      sincosf_core(w, &s2, &c2);
      bad[4] += diff(s1, s2) + diff(c1, c2);
    }
    const float bb = i % 3 ? asfloat((asuint(a) & 0x7f800000u) | (asuint(b) & 0x807fffffu)) : b;
    if (atan2f_ok(a, bb)) {
      bool no = false;
      const float r = atan2f_core(a, bb, &no);
      if (!no) bad[5] += diff(r, dm::atan2f(a, bb));
    }
    const float c = asfloat((static_cast<uint32_t>(v) & 0x7fffffu) | (107u + (v >> 33) % 41u) << 23);
    bad[6] += diff(pt::div_by(any, c, 1.0f / c), any / c);
  }
}

}  // extern "C"
