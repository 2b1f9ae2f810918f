// SPH derivatives, mixed-precision form.
//
// Same physics as SPHHydroBase::evaluateDerivatives
// (src/SPH/SPHHydroBase.cc:471-928) with the pair arithmetic in FP32:
//   - relative position and velocity are formed in FP64 and rounded once;
//   - table kernel, gradient, Monaghan-Gingold Pi and pressure terms in FP32
//     (hardware rsqrt / reciprocal through __frsqrt_rn / __fdividef);
//   - per-node sums in FP32 with Kahan compensation;
//   - the per-node finish (3x3 M inverse, ideal H) and everything outside the
//     pair loop stay FP64.
// Pair terms are formed from node i's side (r_ij = r_i - r_j); every term of
// the reference is odd in r_ij and v_ij or even in both, so the i-side form
// equals the owner-side form up to rounding.  The stored pair accelerations
// are flipped to owner orientation for the compatible-energy update.
#include "problem.cuh"
#include "mixed.cuh"

namespace sphgpu {

namespace {

struct Kahan {
  float s, c;
  __device__ __forceinline__ void init() { s = 0.0f; c = 0.0f; }
  __device__ __forceinline__ void add(float x) {
    const float y = x - c;
    const float t = s + y;
    c = (t - s) - y;
    s = t;
  }
  __device__ __forceinline__ double value() const { return (double)s - (double)c; }
};

struct MRec {
  double x, y, z, vx, vy, vz;
  float m, rho, cs, Hdet, hxx, hxy, hxz, hyy, hyz, hzz, Prho, mrho, P, somega;
  float iso;           // 1: H = hxx I (the symmetric products reduce to scalings)
};

__device__ __forceinline__ MRec loadMRec(const double* mrec, int64_t cap, int64_t k) {
  double a[MRECW];
  ldPlanes<MRECW/4, true>(mrec, cap, k, a);
  MRec R;
  // the layout of writeMixedRecord (problem.cuh)
  R.x = a[0]; R.y = a[1]; R.z = a[2]; R.vx = a[3]; R.vy = a[4]; R.vz = a[5];
  R.m = loF(a[6]); R.rho = hiF(a[6]); R.cs = loF(a[7]); R.Hdet = hiF(a[7]);
  R.hxx = loF(a[8]); R.hxy = hiF(a[8]); R.hxz = loF(a[9]); R.hyy = hiF(a[9]);
  R.hyz = loF(a[10]); R.hzz = hiF(a[10]); R.Prho = loF(a[11]); R.mrho = hiF(a[11]);
  R.P = loF(a[12]); R.somega = hiF(a[12]); R.iso = loF(a[13]);
  return R;
}

__global__ void table_to_float_kernel(const double* coef, int n, float* out) {
  for (int t = blockIdx.x*blockDim.x + threadIdx.x; t < 6*n; t += gridDim.x*blockDim.x) out[t] = (float)coef[t];
}

struct F3 {
  float x, y, z;
};
__device__ __forceinline__ F3 symdot(float xx, float xy, float xz, float yy, float yz, float zz, const F3& r) {
  return F3{xx*r.x + xy*r.y + xz*r.z, xy*r.x + yy*r.y + yz*r.z, xz*r.x + yz*r.y + zz*r.z};
}

__device__ __forceinline__ void tableF(const float* coef, int n, float invStep, float extent, float eta, float Hdet,
                                       float& W, float& gW) {
  if (eta < extent) {
    const float q = eta*invStep;
    int lb = (int)q;
    lb = lb < n - 1 ? lb : n - 1;
    const int i0 = lb < n - 3 ? lb : n - 3;
    const float x = q - (float)i0;
    const float2* c = reinterpret_cast<const float2*>(coef + 6*(i0 + 1));
    const float2 c01 = __ldg(c), c23 = __ldg(c + 1), c45 = __ldg(c + 2);
    W = Hdet*(c01.x + x*(c01.y + x*c23.x));
    gW = Hdet*(c23.y + x*(c45.x + x*c45.y));
  } else {
    W = 0.0f;
    gW = 0.0f;
  }
}

// The sums of a node's row, in the order of the terms below.
enum MSum {
  MS_WNS = 0, MS_M2 = 1, MS_RHO = 7, MS_NORM = 8, MS_EFFVP = 9, MS_VISCW = 10, MS_DVDT = 11, MS_DEPSDT = 14,
  MS_DVDX = 15, MS_M = 24, MS_XSPHW = 33, MS_XSPHDV = 34, MS_ALL = 37
};

// Scalars of the pair arithmetic, rounded once.
struct MConst {
  const float* coef;
  int nt;
  float invStep, extent, eps2, Cl, Cq;
};
__device__ __forceinline__ MConst mixedConst(const Member& MB) {
  const Params& P = MB.prm;
  return MConst{MB.coefF, P.W.n, (float)(1.0/P.W.stepSize), (float)P.W.extent, (float)P.eps2, (float)P.Cl, (float)P.Cq};
}

// The terms of the directed pair (i, j) that node i's sums take: t[MSum], the
// viscous pressure Qi (a maximum) and the pair's acceleration dd.  fs: the
// Balsara shear correction of the pair (max of the two nodes'), else 1.
template<bool XSPH, bool TENSILE>
__device__ __forceinline__ void mixedTerms(const MRec& I, const MRec& J, bool own, const Params& P, const MConst& C,
                                           float fs, float* t, float& Qi, F3& dd) {
  const float ClP = C.Cl*fs, CqP = C.Cq*fs;
  // FP64 differences, rounded once
  const F3 rij{(float)(I.x - J.x), (float)(I.y - J.y), (float)(I.z - J.z)};
  const F3 vij{(float)(I.vx - J.vx), (float)(I.vy - J.vy), (float)(I.vz - J.vz)};
  // isotropic H (the common case): H r = hxx r, bit-identical to the full product
  const bool isoPair = I.iso != 0.0f && J.iso != 0.0f;
  F3 etai, etaj;
  if (isoPair) {
    etai = F3{I.hxx*rij.x, I.hxx*rij.y, I.hxx*rij.z};
    etaj = F3{J.hxx*rij.x, J.hxx*rij.y, J.hxx*rij.z};
  } else {
    etai = symdot(I.hxx, I.hxy, I.hxz, I.hyy, I.hyz, I.hzz, rij);
    etaj = symdot(J.hxx, J.hxy, J.hxz, J.hyy, J.hyz, J.hzz, rij);
  }
  const float e2i = etai.x*etai.x + etai.y*etai.y + etai.z*etai.z;
  const float e2j = etaj.x*etaj.x + etaj.y*etaj.y + etaj.z*etaj.z;
  const float rinvi = e2i > 0.0f ? __frsqrt_rn(e2i) : 0.0f;
  const float rinvj = e2j > 0.0f ? __frsqrt_rn(e2j) : 0.0f;
  const float etaMagi = e2i*rinvi, etaMagj = e2j*rinvj;
  const F3 ui = e2i > 0.0f ? F3{etai.x*rinvi, etai.y*rinvi, etai.z*rinvi} : F3{1.0f, 0.0f, 0.0f};
  const F3 uj = e2j > 0.0f ? F3{etaj.x*rinvj, etaj.y*rinvj, etaj.z*rinvj} : F3{1.0f, 0.0f, 0.0f};
  F3 Hetai, Hetaj;
  if (isoPair) {
    Hetai = F3{I.hxx*ui.x, I.hxx*ui.y, I.hxx*ui.z};
    Hetaj = F3{J.hxx*uj.x, J.hxx*uj.y, J.hxx*uj.z};
  } else {
    Hetai = symdot(I.hxx, I.hxy, I.hxz, I.hyy, I.hyz, I.hzz, ui);
    Hetaj = symdot(J.hxx, J.hxy, J.hxz, J.hyy, J.hyz, J.hzz, uj);
  }
  float Wi, gWi, Wj, gWj;
  tableF(C.coef, C.nt, C.invStep, C.extent, etaMagi, I.Hdet, Wi, gWi);
  tableF(C.coef, C.nt, C.invStep, C.extent, etaMagj, J.Hdet, Wj, gWj);
  const F3 gradWi{Hetai.x*gWi, Hetai.y*gWi, Hetai.z*gWi};
  const F3 gradWj{Hetaj.x*gWj, Hetaj.y*gWj, Hetaj.z*gWj};

  const float rij2 = rij.x*rij.x + rij.y*rij.y + rij.z*rij.z;
  const float r6 = rij2*rij2*rij2;
  const float thptS = r6 > 1.0e-30f ? __fdividef(1.0f, r6) : 1.0e30f;
  t[MS_WNS] = fabsf(gWi);
  const float g2 = (gradWi.x*gradWi.x + gradWi.y*gradWi.y + gradWi.z*gradWi.z)*thptS;
  t[MS_M2 + 0] = rij.x*rij.x*g2; t[MS_M2 + 1] = rij.x*rij.y*g2; t[MS_M2 + 2] = rij.x*rij.z*g2;
  t[MS_M2 + 3] = rij.y*rij.y*g2; t[MS_M2 + 4] = rij.y*rij.z*g2; t[MS_M2 + 5] = rij.z*rij.z*g2;
  t[MS_RHO] = J.m*Wi;
  t[MS_NORM] = I.mrho*Wi;

  // Monaghan-Gingold Pi
  const float mui = __fdividef(vij.x*etai.x + vij.y*etai.y + vij.z*etai.z, e2i + C.eps2);
  const float muj = __fdividef(vij.x*etaj.x + vij.y*etaj.y + vij.z*etaj.z, e2j + C.eps2);
  const float mi0 = fminf(0.0f, mui), mj0 = fminf(0.0f, muj);
  const float ei = -ClP*I.cs*(P.linearInExp ? mui : mi0) + CqP*(P.quadInExp ? -copysignf(1.0f, mui)*mui*mui : mi0*mi0);
  const float ej = -ClP*J.cs*(P.linearInExp ? muj : mj0) + CqP*(P.quadInExp ? -copysignf(1.0f, muj)*muj*muj : mj0*mj0);
  const float qi = __fdividef(ei, I.rho), qj = __fdividef(ej, J.rho);
  const F3 Qacci{0.5f*qi*gradWi.x, 0.5f*qi*gradWi.y, 0.5f*qi*gradWi.z};
  const F3 Qaccj{0.5f*qj*gradWj.x, 0.5f*qj*gradWj.y, 0.5f*qj*gradWj.z};
  const float workQi = vij.x*Qacci.x + vij.y*Qacci.y + vij.z*Qacci.z;
  Qi = I.rho*I.rho*fabsf(qi);
  t[MS_EFFVP] = J.mrho*Qi*Wi;
  t[MS_VISCW] = J.m*workQi;

  float Prhoi = I.Prho, Prhoj = J.Prho;
  if (TENSILE) {
    const float Wo = own ? Wi : Wj, Hdo = own ? I.Hdet : J.Hdet;
    const float x = __fdividef(Wo, Hdo*(float)P.WnPerh);
    const float fij = (float)P.epsTensile*(x*x*x*x);
    Prhoi = __fdividef(I.somega*(I.P + fij*(I.P < 0.0f ? -I.P : 0.0f)), I.rho*I.rho);
    Prhoj = __fdividef(J.somega*(J.P + fij*(J.P < 0.0f ? -J.P : 0.0f)), J.rho*J.rho);
  }
  dd = F3{Prhoi*gradWi.x + Prhoj*gradWj.x + Qacci.x + Qaccj.x,
          Prhoi*gradWi.y + Prhoj*gradWj.y + Qacci.y + Qaccj.y,
          Prhoi*gradWi.z + Prhoj*gradWj.z + Qacci.z + Qaccj.z};
  t[MS_DVDT + 0] = -J.m*dd.x; t[MS_DVDT + 1] = -J.m*dd.y; t[MS_DVDT + 2] = -J.m*dd.z;
  t[MS_DEPSDT] = J.m*(Prhoi*(vij.x*gradWi.x + vij.y*gradWi.y + vij.z*gradWi.z) + workQi);
  const float mj = J.m;
  const F3 mg{mj*gradWi.x, mj*gradWi.y, mj*gradWi.z};
  const float v[3] = {vij.x, vij.y, vij.z}, r[3] = {rij.x, rij.y, rij.z}, g[3] = {mg.x, mg.y, mg.z};
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      t[MS_DVDX + 3*a + c] = -v[a]*g[c];
      t[MS_M + 3*a + c] = -r[a]*g[c];
    }
  if (XSPH) {
    const float w = 0.5f*(I.mrho*Wi + J.mrho*Wj);
    t[MS_XSPHW] = w;
    t[MS_XSPHDV + 0] = -w*vij.x; t[MS_XSPHDV + 1] = -w*vij.y; t[MS_XSPHDV + 2] = -w*vij.z;
  }
}

// the owner's pair acceleration, -m_other*deltaDvDt in owner orientation
// (FP32 in the mixed form; both nodes of the pair read the same value)
__device__ __forceinline__ void storePairAcc(double* pacc, int64_t ecap, int64_t k, bool own, float mi, float mj,
                                             const F3& dd) {
  const float s = own ? -mj : mi;
  float* pf = reinterpret_cast<float*>(pacc);
  pf[k] = s*dd.x;
  pf[ecap + k] = s*dd.y;
  pf[2*ecap + k] = s*dd.z;
}

// The per-node finish in FP64 (src/SPH/SPHHydroBase.cc:834-902) from the sums
// F[MSum] and the stores of the node's derivatives.  midInS0: the RK2 step's
// record-only mid point ran (update_kernel recordMid): the FP64 mid-point H
// and mass density of a member without grad-h are in S0, S holds the start of
// the step.  vi: the node's (mid-point) velocity.
template<bool XSPH>
__device__ __forceinline__ void finishMixed(const Member& MB, int64_t i, const V3& vi, const double* F, float maxvp,
                                            int midInS0) {
  const Params& P = MB.prm;
  const int64_t n = MB.n;
  const double* S = MB.S;
  // exact FP64 node values for the finish
  const double* Sm = midInS0 && !P.gradh && !P.balsara ? MB.S0 : S;
  const Sym Hi{Sm[(S_H + 0)*n + i], Sm[(S_H + 1)*n + i], Sm[(S_H + 2)*n + i],
               Sm[(S_H + 3)*n + i], Sm[(S_H + 4)*n + i], Sm[(S_H + 5)*n + i]};
  const double mi = S[S_M*n + i], rhoi = Sm[S_RHO*n + i], Hdeti = sdet(Hi);
  const int numNeighbors = (int)(MB.offsets[i + 1] - MB.offsets[i]);
  double rhoS = F[MS_RHO] + mi*P.W0*Hdeti;
  double nrm = F[MS_NORM] + mi/rhoi*P.W0*Hdeti;
  T9 Mi{F[MS_M], F[MS_M + 1], F[MS_M + 2], F[MS_M + 3], F[MS_M + 4], F[MS_M + 5], F[MS_M + 6], F[MS_M + 7], F[MS_M + 8]};
  T9 DvDxi{F[MS_DVDX], F[MS_DVDX + 1], F[MS_DVDX + 2], F[MS_DVDX + 3], F[MS_DVDX + 4], F[MS_DVDX + 5],
           F[MS_DVDX + 6], F[MS_DVDX + 7], F[MS_DVDX + 8]};
  if (P.correctVelGrad && fabs(tdet(Mi)) > 1.0e-10 && numNeighbors > 8) {
    Mi = tinverse(Mi);
    DvDxi = tdot(DvDxi, Mi);
  } else {
    DvDxi = tdiv(DvDxi, rhoi);
  }
  const double DrhoDt = -rhoi*ttrace(DvDxi);
  double w = dmax(0.0, F[MS_WNS]/Hdeti);
  w = cbrt(w);
  Sym m2s{F[MS_M2], F[MS_M2 + 1], F[MS_M2 + 2], F[MS_M2 + 3], F[MS_M2 + 4], F[MS_M2 + 5]};
  m2s = sdiv(m2s, Hdeti*Hdeti);
  V3 DxDt = vi;
  double xw = 0.0;
  V3 xdv{0.0, 0.0, 0.0};
  if (XSPH) {
    xw = F[MS_XSPHW];
    xdv = V3{F[MS_XSPHDV], F[MS_XSPHDV + 1], F[MS_XSPHDV + 2]};
    xw += Hdeti*mi/rhoi*P.W0;
    DxDt = vadd(vi, vdiv(xdv, dmax(1.0e-30, xw)));
  }
  const Sym DHDt = smul(sdiv(sneg(Hi), 3.0), ttrace(DvDxi));
  double nPerhCur;
  if (fuzzyEqual(w, 0.0)) {
    nPerhCur = 0.5*P.nPerh;
  } else {
    nPerhCur = equivalentNodesPerSmoothingScale(P, w);
  }
  const double s = dmin(4.0, dmax(0.25, P.nPerh/(nPerhCur + 1.0e-30)));
  const double a = s < 1.0 ? 0.4*(1.0 + s*s) : 0.4*(1.0 + 1.0/(s*s*s));
  const double hi1 = dmin(P.hmax, dmax(P.hmin, (1.0/Hi.xx)*(1.0 - a + a*s)));
  const double hinv = 1.0/hi1;

  double* d = MB.D + i;
  d[(D_DXDT + 0)*n] = DxDt.x; d[(D_DXDT + 1)*n] = DxDt.y; d[(D_DXDT + 2)*n] = DxDt.z;
  d[(D_DVDT + 0)*n] = F[MS_DVDT]; d[(D_DVDT + 1)*n] = F[MS_DVDT + 1]; d[(D_DVDT + 2)*n] = F[MS_DVDT + 2];
  d[D_DRHODT*n] = DrhoDt;
  d[D_DEPSDT*n] = F[MS_DEPSDT];
  d[(D_DHDT + 0)*n] = DHDt.xx; d[(D_DHDT + 1)*n] = DHDt.xy; d[(D_DHDT + 2)*n] = DHDt.xz;
  d[(D_DHDT + 3)*n] = DHDt.yy; d[(D_DHDT + 4)*n] = DHDt.yz; d[(D_DHDT + 5)*n] = DHDt.zz;
  d[(D_HIDEAL + 0)*n] = hinv; d[(D_HIDEAL + 1)*n] = 0.0; d[(D_HIDEAL + 2)*n] = 0.0;
  d[(D_HIDEAL + 3)*n] = hinv; d[(D_HIDEAL + 4)*n] = 0.0; d[(D_HIDEAL + 5)*n] = hinv;
  const double* dv = &DvDxi.xx;
  const double* mm = &Mi.xx;
#pragma unroll
  for (int c = 0; c < 9; ++c) {
    d[(D_DVDX + c)*n] = dv[c];
    d[(D_M + c)*n] = mm[c];
  }
  d[D_RHOSUM*n] = rhoS;
  d[D_NORM*n] = nrm;
  d[D_WNS*n] = w;
  d[(D_M2 + 0)*n] = m2s.xx; d[(D_M2 + 1)*n] = m2s.xy; d[(D_M2 + 2)*n] = m2s.xz;
  d[(D_M2 + 3)*n] = m2s.yy; d[(D_M2 + 4)*n] = m2s.yz; d[(D_M2 + 5)*n] = m2s.zz;
  d[D_XSPHW*n] = xw;
  d[(D_XSPHDV + 0)*n] = xdv.x; d[(D_XSPHDV + 1)*n] = xdv.y; d[(D_XSPHDV + 2)*n] = xdv.z;
  d[D_MAXVP*n] = (double)maxvp;
  d[D_EFFVP*n] = F[MS_EFFVP];
  d[D_VISCW*n] = F[MS_VISCW];
}

// SPHHydroBase::evaluateDerivatives, mixed form: one thread per internal node.
template<bool XSPH, bool TENSILE, bool COMPAT, bool SOLO, bool BALSARA>
__global__ void __launch_bounds__(128, SPH_MIXED_MIN_BLOCKS) sph_eval_mixed_kernel(const Member* mem, BlockMap bm, const Member single,
                                                                 int midInS0) {
  constexpr int NS = XSPH ? MS_ALL : MS_XSPHW;
  const MemberBlock mb = memberBlock(bm);
  const Member& MB = SOLO ? single : mem[mb.m];   // one member: read from the kernel parameters
  const int64_t n = MB.n;
  const int64_t i = mb.block*blockDim.x + threadIdx.x;
  if (i >= n) return;
  const Params& P = MB.prm;
  const MConst C = mixedConst(MB);
  const double* mrec = MB.mrec;
  const int64_t cap = MB.candcap;
  const int32_t* nbr = MB.nbr;
  const MRec I = loadMRec(mrec, cap, i);
  Kahan sum[NS];
#pragma unroll
  for (int c = 0; c < NS; ++c) sum[c].init();
  float maxvp = 0.0f;
  const float fsi = BALSARA ? (float)MB.fshear[i] : 1.0f;
  const int64_t k0 = MB.offsets[i], k1 = MB.offsets[i + 1];
  for (int64_t k = k0; k < k1; ++k) {
    const int32_t j = __ldg(nbr + k);
    const MRec J = loadMRec(mrec, cap, j);
    const float fs = BALSARA ? fmaxf(fsi, (float)MB.fshear[j < n ? (int64_t)j : (int64_t)MB.groot[j - n]]) : 1.0f;
    const bool own = j > (int32_t)i;
    float t[NS], Qi;
    F3 dd;
    mixedTerms<XSPH, TENSILE>(I, J, own, P, C, fs, t, Qi, dd);
#pragma unroll
    for (int c = 0; c < NS; ++c) sum[c].add(t[c]);
    maxvp = fmaxf(maxvp, Qi);
    if (COMPAT) storePairAcc(MB.pacc, MB.ecap, k, own, I.m, J.m, dd);
  }
  double F[NS];
#pragma unroll
  for (int c = 0; c < NS; ++c) F[c] = sum[c].value();
  finishMixed<XSPH>(MB, i, V3{I.vx, I.vy, I.vz}, F, maxvp, midInS0);
}

// The same with a group of 16 lanes per node, for long rows (the FP64 form's
// sph_eval_fp64_rows_kernel says why): the lanes form the terms of 16 entries,
// then lane l adds those of its sums (l, l + 16, l + 32) in row order.  The
// Kahan sums take the valid entries only (a zero term is not neutral there),
// so every sum has the thread-per-node kernel's bits.
constexpr int kRowLanes = 16;
constexpr int kRowPad = kRowLanes + 1;
constexpr int kRowGroups = 128/kRowLanes;

template<bool XSPH, bool TENSILE, bool COMPAT, bool SOLO, bool BALSARA>
__global__ void __launch_bounds__(128, SPH_MIXED_ROWS_MIN_BLOCKS) sph_eval_mixed_rows_kernel(const Member* mem, BlockMap bm, const Member single,
                                                                      int midInS0, int nodes) {
  constexpr int NS = XSPH ? MS_ALL : MS_XSPHW;
  __shared__ float sT[kRowGroups][(NS + 1)*kRowPad];
  __shared__ double sF[kRowGroups*kRowMaxNodes][NS + (NS + 1) % 2];      // (odd stride: the finish reads a node per thread)
  __shared__ float sQ[kRowGroups*kRowMaxNodes];
  const MemberBlock mb = memberBlock(bm);
  const Member& MB = SOLO ? single : mem[mb.m];
  const int64_t n = MB.n;
  const Params& P = MB.prm;
  const MConst C = mixedConst(MB);
  const double* mrec = MB.mrec;
  const int64_t cap = MB.candcap;
  const int32_t* nbr = MB.nbr;
  const int grp = threadIdx.x/kRowLanes, l = threadIdx.x % kRowLanes;
  const unsigned half = 0xffffu << (threadIdx.x & 16);
  const int64_t first = mb.block*(int64_t)(kRowGroups*nodes);
  float* T = sT[grp];
  for (int q = 0; q < nodes; ++q) {
    const int64_t i = first + q*kRowGroups + grp;
    if (i >= n) break;
    const MRec I = loadMRec(mrec, cap, i);
    const float fsi = BALSARA ? (float)MB.fshear[i] : 1.0f;
    Kahan s0, s1, s2;
    s0.init(); s1.init(); s2.init();
    float maxvp = 0.0f;
    const int64_t k0 = MB.offsets[i], k1 = MB.offsets[i + 1];
    for (int64_t base = k0; base < k1; base += kRowLanes) {
      const int64_t k = base + l;
      if (k < k1) {
        const int32_t j = __ldg(nbr + k);
        const MRec J = loadMRec(mrec, cap, j);
        const float fs = BALSARA ? fmaxf(fsi, (float)MB.fshear[j < n ? (int64_t)j : (int64_t)MB.groot[j - n]]) : 1.0f;
        const bool own = j > (int32_t)i;
        float t[NS], Qi;
        F3 dd;
        mixedTerms<XSPH, TENSILE>(I, J, own, P, C, fs, t, Qi, dd);
#pragma unroll
        for (int c = 0; c < NS; ++c) T[c*kRowPad + l] = t[c];
        maxvp = fmaxf(maxvp, Qi);
        if (COMPAT) storePairAcc(MB.pacc, MB.ecap, k, own, I.m, J.m, dd);
      }
      __syncwarp(half);
      const int valid = k1 - base < kRowLanes ? (int)(k1 - base) : kRowLanes;
      const float* t0 = T + l*kRowPad;
      const float* t1 = t0 + kRowLanes*kRowPad;
      const float* t2 = t1 + (l < NS - 2*kRowLanes ? kRowLanes*kRowPad : 0);   // (a second copy where there is no third sum)
      if (valid == kRowLanes) {
#pragma unroll
        for (int e = 0; e < kRowLanes; ++e) { s0.add(t0[e]); s1.add(t1[e]); s2.add(t2[e]); }
      } else {
        for (int e = 0; e < valid; ++e) { s0.add(t0[e]); s1.add(t1[e]); s2.add(t2[e]); }
      }
      __syncwarp(half);
    }
    for (int o = 8; o > 0; o >>= 1) maxvp = fmaxf(maxvp, __shfl_xor_sync(half, maxvp, o));
    double* F = sF[q*kRowGroups + grp];
    F[l] = s0.value();
    F[l + kRowLanes] = s1.value();
    if (l < NS - 2*kRowLanes) F[l + 2*kRowLanes] = s2.value();
    if (l == 0) sQ[q*kRowGroups + grp] = maxvp;
  }
  __syncthreads();
  // the finish, a thread per node of the block
  const int64_t i = first + threadIdx.x;
  if ((int)threadIdx.x >= kRowGroups*nodes || i >= n) return;
  const D4 xv = ldPlane(mrec + planeAt(cap, i, 0)), v2 = ldPlane(mrec + planeAt(cap, i, 1));
  finishMixed<XSPH>(MB, i, V3{xv.d, v2.a, v2.b}, sF[threadIdx.x], sQ[threadIdx.x], midInS0);
}

}  // namespace

int prepare_mixed(Batch& b) {
  for (Problem* pp : b.mem) {
    Problem& p = *pp;
    if (p.cfg.precision != SPHGPU_PRECISION_MIXED) continue;
    if (p.coefF == nullptr) {
      if (dev_alloc(reinterpret_cast<void**>(&p.coefF), sizeof(float)*6*(size_t)p.prm.W.n) != cudaSuccess) {
        set_error("mixed table allocation failed");
        return SPHGPU_ERR_NOMEM;
      }
      table_to_float_kernel<<<8, 256, 0, b.stream>>>(p.prm.W.coef, p.prm.W.n, p.coefF); ++p.launches;
      b.memDirty = true;
    }
    const int64_t need = p.candcap;
    if (need > p.mreccap) {
      cudaStreamSynchronize(b.stream);
      dev_free(p.mrec);
      p.mrec = nullptr;
      if (dev_alloc(reinterpret_cast<void**>(&p.mrec), sizeof(double)*(p.prm.hydro == SPHGPU_HYDRO_CRKSPH ? CMRECW : MRECW)*(size_t)need) != cudaSuccess) {
        p.mreccap = 0;
        set_error("mixed record allocation failed");
        return SPHGPU_ERR_NOMEM;
      }
      p.mreccap = need;
      b.memDirty = true;
    }
  }
  if (b.memDirty) SPH_TRY(batch_upload(b));
  return SPHGPU_OK;
}

// SPH members in the mixed form (CRKSPH members in the mixed form have their
// own records and kernels, crk_mixed.cu)
bool mixedSph(const Problem& p) {
  return p.cfg.precision == SPHGPU_PRECISION_MIXED && p.prm.hydro == SPHGPU_HYDRO_SPH;
}

// One launch of the mixed pair kernel variant <XSPH, TENSILE, COMPAT, BALSARA>;
// nodes > 0: of the row kernel.
template<bool X, bool T, bool C, bool B>
void launch_mixed_variant(Batch& b, unsigned grid, BlockMap bm, const Member& one, bool solo, int mid, int nodes) {
  if (nodes > 0) {
    if (solo) sph_eval_mixed_rows_kernel<X, T, C, true, B><<<grid, 128, 0, b.stream>>>(b.d_mem, bm, one, mid, nodes);
    else sph_eval_mixed_rows_kernel<X, T, C, false, B><<<grid, 128, 0, b.stream>>>(b.d_mem, bm, one, mid, nodes);
  } else if (solo) {
    sph_eval_mixed_kernel<X, T, C, true, B><<<grid, b.evalThreads, 0, b.stream>>>(b.d_mem, bm, one, mid);
  } else {
    sph_eval_mixed_kernel<X, T, C, false, B><<<grid, b.evalThreads, 0, b.stream>>>(b.d_mem, bm, one, mid);
  }
}
using MixedLaunch = void (*)(Batch&, unsigned, BlockMap, const Member&, bool, int, int);
// indexed by BALSARA << 3 | XSPH << 2 | TENSILE << 1 | COMPAT
const MixedLaunch kMixedLaunch[16] = {
    &launch_mixed_variant<false, false, false, false>, &launch_mixed_variant<false, false, true, false>,
    &launch_mixed_variant<false, true, false, false>, &launch_mixed_variant<false, true, true, false>,
    &launch_mixed_variant<true, false, false, false>, &launch_mixed_variant<true, false, true, false>,
    &launch_mixed_variant<true, true, false, false>, &launch_mixed_variant<true, true, true, false>,
    &launch_mixed_variant<false, false, false, true>, &launch_mixed_variant<false, false, true, true>,
    &launch_mixed_variant<false, true, false, true>, &launch_mixed_variant<false, true, true, true>,
    &launch_mixed_variant<true, false, false, true>, &launch_mixed_variant<true, false, true, true>,
    &launch_mixed_variant<true, true, false, true>, &launch_mixed_variant<true, true, true, true>};

int launch_eval_sph_mixed(Batch& b) {
  auto mixed = mixedSph;
  SPH_TRY(pack_mixed(b, false));
  auto key = [](const Problem& p) {
    return (p.prm.balsara ? 8 : 0) | (p.prm.XSPH ? 4 : 0) | (p.prm.epsTensile != 0.0 ? 2 : 0) |
           (p.prm.compatible ? 1 : 0);
  };
  const bool solo = b.mem.size() == 1;
  const Member one = solo ? describe_member(*b.mem[0]) : Member{};
  const int mid = b.midInS0 ? 1 : 0;
  bool present[16] = {};
  for (Problem* p : b.mem) if (mixed(*p)) present[key(*p)] = true;
  for (int v = 0; v < 32; ++v) {
    const bool rows = (v & 16) != 0;
    if (!present[v & 15]) continue;
    auto mine = [&](const Problem& p) { return mixed(p) && key(p) == (v & 15) && longRows(p) == rows; };
    int64_t total = 0;
    for (Problem* p : b.mem) total += mine(*p) ? p->n : 0;
    if (total == 0) continue;
    const int nodes = rows ? rowNodes(total) : 0;
    BlockMap bm;
    unsigned grid = 0;
    SPH_TRY(batch_map_items(b, [&](const Problem& p) { return mine(p) ? p.n : (int64_t)0; },
                            rows ? kRowGroups*nodes : b.evalThreads, &bm, &grid));
    if (!grid) continue;
    kMixedLaunch[v & 15](b, grid, bm, one, solo, mid, nodes);
    batch_count_launch(b);
  }
  return cuda_status(cudaGetLastError(), "evaluate (mixed)");
}

}  // namespace sphgpu
