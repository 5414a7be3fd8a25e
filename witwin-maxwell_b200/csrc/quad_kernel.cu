// Quad-tile fused leapfrog step (launch variant 11): one launch advances
// H^{n-1/2} -> H^{n+1/2} and E^n -> E^{n+1} over the whole grid, CPML included.
//
// A CTA owns QuadShape::TY whole z rows and marches +x over a chunk of planes.  A
// thread owns one quad: four consecutive z cells of one row, so every field,
// coefficient and psi access is one 16-byte load or store and the per-cell
// instruction count is a quarter of a one-cell-per-lane kernel's.  Whole rows need
// no z halo; one extra row (j0 - 1) of threads recomputes the halo H that the first
// owned row reads and stores nothing.
//
// Data movement: a copy warp brings the rows of the E and H planes (contiguous in
// memory) into a three-slot ring in shared memory with cp.async.bulk, and with them
// the z-slab psi of the plane, which a few warps need and would otherwise wait for.
// Batch u holds E(i + 1), H(i) and psi(i) of plane i = istart + u (batch 0 also
// E(istart)) behind one mbarrier.  Per plane every thread waits for its batch,
// computes H^{n+1/2}(i) of its quad and writes it over H^{n-1/2}(i) in the ring,
// meets one block barrier, and computes E^{n+1}(i) from its own H, the H of the row
// and quad before it (ring) and its H of plane i - 1 (registers).  After the barrier
// of plane i nobody reads E(i) or H(i - 1) again, so those slots take batch u + 2: a
// batch is in flight for one and a half planes, about 90 KB per SM at 256^3, twice
// what one SM needs to keep HBM busy.
//
// Slab and face code runs only in the warps that need it: the first and last quads
// of the rows (z faces and z slabs) are dealt to warps of their own, every branch on
// them is uniform over a warp, and a warp without slab cells runs a march without
// that code (717 -> 560 warp instructions per plane with a 10-cell CPML, 130 ->
// 122 us at 193 x 193 x 161; z-slab psi from the ring instead of from L2: -> 108 us).
//
// What bounds it: without slab code the copies on large grids (257^3, one source: 0.89
// of the measured copy rate; 182 x 212 x 158, less than one round of CTAs: 0.68).
// With it the plane barrier, at which a warp in a slab holds its CTA, 19 warps and
// one CTA per SM (193 x 193 x 161, 10 cells: DRAM at 0.46 of the copy rate, an issue in
// 0.41 of the cycles, the barrier the largest stall).  On small grids the launch and the
// latency of two planes (25 x 21 x 19: 14 us).  See default_quad (engine.cu) for the
// tile rule and the measured times.
//
// Every mbarrier wait is bounded (StepParams::wait_limit polls).  A wait that
// runs out records FDTD_ERR_TIMEOUT in p.status; the thread carries on without
// waiting (its values are garbage, which the status makes the host discard) so
// that every block barrier is still met, and the issuing thread stops copying
// and waits, with its own bound, for the copies in flight before the block ends.
//
// Deferred (wrap-face) cells get a value that the wrap kernel (bloch.cu)
// overwrites; their psi is left alone.  Poles run in the ADE pass (ade_pass.cu).
//
// Products and sums are written with explicit rounding: a warp's body is chosen
// by its class, and every body has to give a cell the same bits (the warp and
// row-tile kernels' bits, but for cells near a slab).
//
// Arithmetic restated from witwin/maxwell/fdtd/cuda/kernels/magnetic.cu:62-212,
// electric.cu:242-311 and 462-941, sources.cu:135-154 and 485-545.
#include "../../include/fdtd_b200.h"
#include "quad_kernel.cuh"
#include "step_device.cuh"

namespace fdtdb200 {

namespace {

constexpr uint32_t kDrainLimit = 1u << 20;  // polls of the final drain
constexpr int kSlots = 3;

__device__ __forceinline__ uint32_t saddr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, uint32_t limit) {
  for (uint32_t it = 0; it < limit; ++it) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// 16-byte aligned global -> shared bulk copy (no multicast).
__device__ __forceinline__ void bulk_load(uint32_t dst, const float* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

// Tile geometry of a CTA.
struct Tile {
  int j0, TY;  // owned rows j0 .. j0 + TY - 1
};

// Copies of one batch by the issuing thread: E plane ie (rows j0 - 1 .. j0 + TY, Ey
// without the last) and H plane ih (rows j0 - 1 .. j0 + TY - 1) with its z-slab psi
// into their slots; a negative plane is skipped.
__device__ __forceinline__ void issue_batch(const StepParams& p, const Tile& t, int ie, int ih, float* es, float* hs,
                                            float* zs, uint32_t bar, int extra_ie, float* extra_es) {
  const int NY = p.NY, P = p.P;
  const int ja = max(t.j0 - 1, 0);
  const int nh = min(t.j0 + t.TY, NY) - ja, ne = min(t.j0 + t.TY + 1, NY) - ja;  // rows
  const uint32_t rowb = 4u * P;
  const int d0 = (ja - (t.j0 - 1)) * P, e_pitch = (t.TY + 2) * P, h_pitch = (t.TY + 1) * P;
  const uint32_t ebytes = rowb * (2 * ne + nh);
  const uint32_t bytes = (ie >= 0 ? ebytes : 0u) + (extra_ie >= 0 ? ebytes : 0u) +
                         (ih >= 0 ? 3u * rowb * nh + 16u * nh * p.SZ : 0u);
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
  const int64_t ps = static_cast<int64_t>(NY) * P, o = static_cast<int64_t>(ja) * P;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const uint32_t eb = rowb * (c == 1 ? nh : ne);
    if (extra_ie >= 0) bulk_load(saddr(extra_es + c * e_pitch + d0), p.Ein[c] + extra_ie * ps + o, eb, bar);
    if (ie >= 0) bulk_load(saddr(es + c * e_pitch + d0), p.Ein[c] + ie * ps + o, eb, bar);
    if (ih >= 0) bulk_load(saddr(hs + c * h_pitch + d0), p.Hin[c] + ih * ps + o, rowb * nh, bar);
  }
  if (p.SZ > 0 && ih >= 0) {
    // whole slab rows of the H terms (Hx, Hy) and the E terms (Ex, Ey)
    const int64_t oz = (static_cast<int64_t>(ih) * NY + ja) * p.SZ;
    const int d = (ja - (t.j0 - 1)) * p.SZ, a = (t.TY + 1) * p.SZ;
    const uint32_t b = 4u * nh * p.SZ;
    bulk_load(saddr(zs + d), p.psiHin[0][1] + oz, b, bar);
    bulk_load(saddr(zs + a + d), p.psiHin[1][1] + oz, b, bar);
    bulk_load(saddr(zs + 2 * a + d), p.psiE[0][1] + oz, b, bar);
    bulk_load(saddr(zs + 3 * a + d), p.psiE[1][1] + oz, b, bar);
  }
}

__device__ __forceinline__ void ld4(float (&v)[4], const float* a) {
  const float4 x = *reinterpret_cast<const float4*>(a);
  v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
}
__device__ __forceinline__ void ldg4(float (&v)[4], const float* a) {
  const float4 x = __ldg(reinterpret_cast<const float4*>(a));
  v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
}
__device__ __forceinline__ void st4(float* a, const float (&v)[4]) {
  *reinterpret_cast<float4*>(a) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void stcg4(float* a, const float (&v)[4]) {
  __stcg(reinterpret_cast<float4*>(a), make_float4(v[0], v[1], v[2], v[3]));
}
__device__ __forceinline__ void fill4(float (&v)[4], float x) { v[0] = v[1] = v[2] = v[3] = x; }

// The cells of a quad on the z faces: cell 0 when `first`, cell `last` (4: none).
struct ZFace {
  bool first;
  int last;
};

// CPML recursion of a quad: psi = b psi + c d, d <- d / kappa + psi, on lanes
// with `act`.  kCd: fold c d into b psi rather than the other way: as the warp kernel
// does, so that both give the same bits.  Cells of `zf` keep their psi (E on a z face is not updated).
template <bool kCd>
__device__ __forceinline__ void psi4z(float (&d)[4], const float (&b)[4], const float (&c)[4], const float (&ik)[4],
                                      const float* in, float* out, bool act, bool write, const ZFace& zf) {
  float s[4], o[4];
  fill4(o, 0.f);
  if (act) ld4(o, in);
#pragma unroll
  for (int q = 0; q < 4; ++q)
    s[q] = kCd ? __fmaf_rn(c[q], d[q], __fmul_rn(b[q], o[q])) : __fmaf_rn(b[q], o[q], __fmul_rn(c[q], d[q]));
#pragma unroll
  for (int q = 0; q < 4; ++q) d[q] = act ? __fmaf_rn(d[q], ik[q], s[q]) : d[q];
  if (zf.first) s[0] = o[0];
#pragma unroll
  for (int q = 0; q < 4; ++q)
    if (q == zf.last) s[q] = o[q];
  if (act && write) st4(out, s);
}
// The same along x or y, where the profile is one value.
template <bool kCd>
__device__ __forceinline__ void psi4(float (&d)[4], const Prof& f, const float* in, float* out, int off, bool act,
                                     bool write, const ZFace& zf) {
  const float b[4] = {f.b, f.b, f.b, f.b}, c[4] = {f.c, f.c, f.c, f.c}, ik[4] = {f.ik, f.ik, f.ik, f.ik};
  psi4z<kCd>(d, b, c, ik, in + off, out + off, act, write, zf);
}
// b, c, 1/kappa of a z-slab quad from the table in shared memory.
__device__ __forceinline__ void ztab(float (&b)[4], float (&c)[4], float (&ik)[4], const float* tab, int SZ) {
  ld4(b, tab);
  ld4(c, tab + SZ);
  ld4(ik, tab + 2 * SZ);
}

// Injection terms `bits` of one phase (component base..base + 2) in plane i on
// the quad at (j, k).
// kTogether: a quad's loads go out together.  One after the other, their latencies make
// a plane with many terms slow (24 dipoles over the same cells of a closed 128^3 box:
// 224 us a step, 182 together; one in 182 x 212 x 158: 62.9 and 59.5).  In the kernels
// with slab code the longer loop costs more than it gives on the thin terms of a TFSF
// box, one cell of a quad each (one channel of the 257 x 257 x 193 grating, z slabs:
// 308 us a step, 315 together).
template <bool kTogether>
__device__ __forceinline__ void quad_terms(const QuadTerms& terms, unsigned bits, int base, int n, int i, int j, int k,
                                           float (&v0)[4], float (&v1)[4], float (&v2)[4]) {
  for (; bits; bits &= bits - 1) {
    const InjectionTerm& t = terms.t[__ffs(bits) - 1];
    if (i < t.i0 || i >= t.i1) continue;
    const int li = i - t.i0, lj = j - t.j0;
    const float* row = t.coeff + (static_cast<int64_t>(li) * (t.j1 - t.j0) + lj) * (t.k1 - t.k0) - t.k0;
    const bool along_z = t.signal == nullptr && t.sample_axis == 2;
    const float* hist = t.aux_hist + static_cast<int64_t>(n) * t.aux_len;
    const int c = t.comp - base;
    if constexpr (kTogether) {
      bool in[4];
      float w[4], s[4];
      const float one = t.signal != nullptr ? __ldg(t.signal + n)
                        : along_z           ? 0.f
                                            : __ldg(hist + __ldg(t.sample_index + (t.sample_axis == 0 ? li : lj)));
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        in[q] = k + q >= t.k0 && k + q < t.k1;
        w[q] = in[q] ? __ldg(row + k + q) : 0.f;
        s[q] = one;
      }
      if (along_z) {
#pragma unroll
        for (int q = 0; q < 4; ++q) s[q] = in[q] ? __ldg(hist + __ldg(t.sample_index + k + q - t.k0)) : 0.f;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float val = __fmul_rn(w[q], s[q]);
        if (c == 0) v0[q] = in[q] ? __fmaf_rn(val, t.scale, v0[q]) : v0[q];
        else if (c == 1) v1[q] = in[q] ? __fmaf_rn(val, t.scale, v1[q]) : v1[q];
        else v2[q] = in[q] ? __fmaf_rn(val, t.scale, v2[q]) : v2[q];
      }
      continue;
    }
    float s = 0.f;
    if (t.signal != nullptr) s = __ldg(t.signal + n);
    else if (!along_z) s = __ldg(hist + __ldg(t.sample_index + (t.sample_axis == 0 ? li : lj)));
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int kk = k + q;
      if (kk < t.k0 || kk >= t.k1) continue;
      if (along_z) s = __ldg(hist + __ldg(t.sample_index + kk - t.k0));
      const float val = __fmul_rn(__ldg(row + kk), s);
      if (c == 0) v0[q] = __fmaf_rn(val, t.scale, v0[q]);
      else if (c == 1) v1[q] = __fmaf_rn(val, t.scale, v1[q]);
      else v2[q] = __fmaf_rn(val, t.scale, v2[q]);
    }
  }
}

// One block barrier per plane.  Warps of different classes meet it from their
// own copy of the march, so it is the bare instruction.
__device__ __forceinline__ void plane_sync() { asm volatile("bar.sync 0;" ::: "memory"); }

// The copy warp: its first lane issues the bulk copies.  It waits for each batch
// like the others, so that it stops issuing when one never lands.
__device__ __forceinline__ void copy_march(const StepParams& p, const Tile& t, float* ering, float* hring, float* zring,
                                           int es, int hs, int zs, uint32_t bar0, int istart, int i1, int lane) {
  int issued = min(2, i1 - istart);
  if (lane == 0) {
    for (int u = 0; u < issued; ++u) {
      const int i = istart + u;
      issue_batch(p, t, i + 1 < p.NX ? i + 1 : -1, i, ering + (u + 1) * es, hring + u * hs, zring + u * zs,
                  bar0 + 8u * u, u == 0 ? istart : -1, ering);
    }
  }
  bool ok = true;
  int sl = 0;
  uint32_t par = 0;
  for (int i = istart; i < i1; ++i) {
    if (lane == 0 && ok) ok = mbar_wait(bar0 + 8u * sl, par, static_cast<uint32_t>(p.wait_limit));
    __syncwarp();
    plane_sync();
    if (lane == 0 && ok && i + 2 < i1) {
      // E(i + 3) over E(i), H(i + 2) over H(i - 1)
      const int prev = sl == 0 ? kSlots - 1 : sl - 1;
      issue_batch(p, t, i + 3 < p.NX ? i + 3 : -1, i + 2, ering + sl * es, hring + prev * hs, zring + prev * zs,
                  bar0 + 8u * prev, -1, nullptr);
      ++issued;
    }
    sl = sl == kSlots - 1 ? 0 : sl + 1;
    if (sl == 0) par ^= 1u;
  }
  // after a wait that ran out, its batch and the one after it may still be in
  // flight: this thread outlives them
  if (lane == 0 && !ok)
    for (int u = max(0, issued - 2); u < issued; ++u)
      mbar_wait(bar0 + 8u * (u % kSlots), (u / kSlots) & 1, kDrainLimit);
}

// Flags of a thread's quad (and, or-ed over the warp, of the warp).
constexpr unsigned kZLast = 7u, kZFirst = 1u << 3, kValid = 1u << 4, kOwn = 1u << 5, kYFace = 1u << 6, kYLast = 1u << 7,
                   kYPec = 1u << 8, kYSlabH = 1u << 9, kYSlabE = 1u << 10, kZSlabH = 1u << 11, kZSlabE = 1u << 12,
                   kWarpZFace = 1u << 13, kWarpECoef = 1u << 14, kWarpHCoef = 1u << 15, kItem = 1u << 16;
constexpr unsigned kYSlab = kYSlabH | kYSlabE, kZSlab = kZSlabH | kZSlabE;

// Offset of a row's y-slab psi (row 0 of the slab where the row has none).
__device__ __forceinline__ int yoff(const StepParams& p, int i, int j, int k, int extent) {
  return yslab_off(p, i, max(slab_coord(p, 1, j, extent), 0), k);
}

// A thread's quad and its CTA's ring.
struct Quad {
  int j, k, jc;      // row, first z cell, row clamped into the grid
  unsigned fl, wf;   // flags of the quad, or-ed over the warp
  unsigned fold;     // cells that fold outside the x blocks of a slab
  unsigned tmask;    // injection terms that meet the quad in some plane of the chunk
  int so;            // own quad inside an E or H component tile
  int istart, i0, i1;
  int e_pitch, h_pitch;
  float* ering;
  float* hring;
  const float* zring;   // own quad in the z-slab psi of slot 0 (slab quads)
  const float* ztable;  // own column of the z tables (slab quads)
  int zs, za;           // sizes of a slot and of an array in it
  uint32_t bar0;
};

// The march of one warp.  kCpml: some quad of the warp lies in a slab in some
// plane of the chunk.  kCoef: some coefficient of its quads differs from the
// background scalar.
// Rounding: an H cell folds the first product of its curl into the difference
// unless a slab meets its row or the row before, its 30-cell z block or its block
// of StepParams::fold_cx planes, and E never folds: the warp kernel's bits, whose
// class bodies the compiler contracts that way (to a few cells at the class
// borders).  kFold: the scene has no CPML; H and E fold, as in the row-tile kernel.
template <bool kCpml, bool kCoef, bool kUniform, bool kFold>
__device__ __forceinline__ void quad_march(const StepParams& p, const QuadTerms& terms, const Quad& c, int n) {
  const int NX = p.NX, NY = p.NY, P = p.P;
  const int j = c.j, k = c.k, jc = c.jc, i0 = c.i0, i1 = c.i1, istart = c.istart;
  const unsigned fl = c.fl, wf = c.wf, tmask = c.tmask;
  const int so = c.so, e_pitch = c.e_pitch, h_pitch = c.h_pitch, es = 3 * e_pitch, hs = 3 * h_pitch;
  float* const ering = c.ering;
  float* const hring = c.hring;
  const uint32_t bar0 = c.bar0;
  const float ihy = kUniform ? p.inv_h_u[1] : __ldg(p.inv_h[1] + min(jc, NY - 2));
  const float iey = kUniform ? p.inv_e_u[1] : __ldg(p.inv_e[1] + jc);
  const int ps = NY * P;
  int o = (istart * NY + jc) * P + k;  // field offset
  auto fold = [](float u, float iu, float v, float iv) { return __fmaf_rn(u, iu, -__fmul_rn(v, iv)); };

  float hpz[4], hpy[4];  // Hz, Hy of plane i - 1
  fill4(hpz, 0.f);
  fill4(hpy, 0.f);
  bool ok = true;
  int se = 0;          // slot of E(i) and H(i)
  uint32_t par = 0;    // parity of the batch of plane i
  for (int i = istart; i < i1; ++i) {
    const bool own = i >= i0;
    const int sen = se == kSlots - 1 ? 0 : se + 1;
    const bool xface = i == 0 || i == NX - 1;
    unsigned fm = 0;  // cells of the quad that fold
    if (!kFold) {
      const int x0 = i - i % p.fold_cx;
      const bool xslab = max(x0 - 1, 0) < p.slab_lo[0] ||
                         (p.slab_hi[0] > 0 && min(x0 + p.fold_cx, NX) - 1 >= NX - 1 - p.slab_hi[0]);
      fm = xslab ? 0u : c.fold;
    }
    const int sxh = kCpml ? slab_coord(p, 0, i, NX - 1) : -1;
    const int sxe = kCpml && !xface ? slab_coord(p, 0, i, NX) : -1;
    if (kCpml && i + 1 < i1) {
      // L2 prefetch of the psi that the next plane reads
      if (sxh >= 0 && (fl & kValid) && slab_coord(p, 0, i + 1, NX - 1) >= 0) {
        const int x = xslab_off(p, sxh + 1, jc, k);
        pf_l2<float>(p.psiHin[1][0], x);
        pf_l2<float>(p.psiHin[2][0], x);
      }
      if (sxe >= 0 && (fl & kOwn) && slab_coord(p, 0, i + 1, NX) >= 0) {
        const int x = xslab_off(p, sxe + 1, jc, k);
        pf_l2<float>(p.psiE[1][0], x);
        pf_l2<float>(p.psiE[2][0], x);
      }
      if (wf & kYSlab) {
        if (fl & kYSlabH) {
          const int x = yoff(p, i + 1, jc, k, NY - 1);
          pf_l2<float>(p.psiHin[0][0], x);
          pf_l2<float>(p.psiHin[2][1], x);
        }
        if (fl & kYSlabE) {
          const int x = yoff(p, i + 1, jc, k, NY);
          pf_l2<float>(p.psiE[0][0], x);
          pf_l2<float>(p.psiE[2][1], x);
        }
      }
    }
    if (kCoef && (wf & kWarpECoef) && i + 1 < i1) {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        if (p.ecurl[c]) pf_l2<float>(p.ecurl[c], o + ps);
        if (p.edecay[c]) pf_l2<float>(p.edecay[c], o + ps);
      }
    }
    if (ok && !mbar_wait(bar0 + 8u * se, par, static_cast<uint32_t>(p.wait_limit))) {
      ok = false;
      atomicExch(p.status, FDTD_ERR_TIMEOUT);
    }
    // ---------------- H^{n+1/2}(i) ----------------
    // Hx: dEz/dy - dEy/dz; Hy: dEx/dz - dEz/dx; Hz: dEy/dx - dEx/dy
    float e0[4], e1[4], e2[4], hx[4], hy[4], hz[4];
    float* hown = hring + se * hs + so;
    const float* zq = c.zring + se * c.zs;
    {
      const bool wr = own && (fl & kOwn);
      const ZFace none{false, 4};
      const float* ec = ering + se * es + so;
      const float* en = ering + sen * es + so;
      ld4(e0, ec);
      ld4(e1, ec + e_pitch);
      ld4(e2, ec + 2 * e_pitch);
      const float ihx = kUniform ? p.inv_h_u[0] : __ldg(p.inv_h[0] + min(i, NX - 2));
      float wz[4], zb[4], zc[4], zik[4], a[4], b[4], w[4], f[4];
      if (kUniform) fill4(wz, p.inv_h_u[2]);
      else ldg4(wz, p.ztab_h + 3 * P + k);
      Prof fx{0.f, 0.f, 1.f}, fy{0.f, 0.f, 1.f};
      if (kCpml) {
        if (sxh >= 0) fx = prof(p.hb[0], p.hc[0], p.hik[0], i);
        if ((wf & kYSlab) && (fl & kYSlabH)) fy = prof(p.hb[1], p.hc[1], p.hik[1], j);
      }
// H = decay H - curl (U - V), U and V the two terms u iu, v iv of the curl; f is
// the difference with the first product folded in.
#define FDTD_QUAD_SCALE(U, IU, V, IV)                                                       \
  do {                                                                                      \
    _Pragma("unroll") for (int q = 0; q < 4; ++q) {                                         \
      f[q] = fold(U[q], IU, V[q], IV);                                                      \
      U[q] = __fmul_rn(U[q], IU);                                                           \
      V[q] = __fmul_rn(V[q], IV);                                                           \
    }                                                                                       \
  } while (0)
#define FDTD_QUAD_H(I, H, U, IU, V, IV)                                                     \
  do {                                                                                      \
    ld4(H, hown + I * h_pitch);                                                             \
    float d[4], c[4];                                                                       \
    fill4(d, p.hdecay_u[I]);                                                                \
    fill4(c, p.hcurl_u[I]);                                                                 \
    if (kCoef && (wf & kWarpHCoef)) {                                                       \
      if (p.hdecay[I]) ldg4(d, p.hdecay[I] + o);                                            \
      if (p.hcurl[I]) ldg4(c, p.hcurl[I] + o);                                              \
    }                                                                                       \
    _Pragma("unroll") for (int q = 0; q < 4; ++q) {                                         \
      const float x = kFold ? fold(U[q], IU, V[q], IV) : ((fm >> q) & 1u ? f[q] : U[q] - V[q]); \
      H[q] = __fmaf_rn(H[q], d[q], -__fmul_rn(c[q], x));                                    \
    }                                                                                       \
  } while (0)
      // Hx
      const float e1k = ec[e_pitch + 4];
      ld4(w, ec + 2 * e_pitch + P);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        a[q] = w[q] - e2[q];
        b[q] = (q < 3 ? e1[q < 3 ? q + 1 : 3] : e1k) - e1[q];
      }
      if (!kFold) FDTD_QUAD_SCALE(a, ihy, b, wz[q]);
      if (kCpml) {
        if (wf & kYSlab)
          psi4<false>(a, fy, p.psiHin[0][0], p.psiHout[0][0], yoff(p, i, jc, k, NY - 1), fl & kYSlabH, wr, none);
        if (wf & kZSlab) {
          ztab(zb, zc, zik, c.ztable, p.SZ);
          psi4z<false>(b, zb, zc, zik, zq, p.psiHout[0][1] + zslab_off(p, i, jc, k), fl & kZSlabH, wr, none);
        }
      }
      FDTD_QUAD_H(0, hx, a, ihy, b, wz[q]);
      // Hy
      const float e0k = ec[4];
      ld4(w, en + 2 * e_pitch);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        a[q] = w[q] - e2[q];
        b[q] = (q < 3 ? e0[q < 3 ? q + 1 : 3] : e0k) - e0[q];
      }
      if (!kFold) FDTD_QUAD_SCALE(b, wz[q], a, ihx);
      if (kCpml) {
        if (sxh >= 0)
          psi4<false>(a, fx, p.psiHin[1][0], p.psiHout[1][0], xslab_off(p, sxh, jc, k), fl & kValid, wr, none);
        if (wf & kZSlab) {
          ztab(zb, zc, zik, c.ztable, p.SZ);
          psi4z<false>(b, zb, zc, zik, zq + c.za, p.psiHout[1][1] + zslab_off(p, i, jc, k), fl & kZSlabH, wr, none);
        }
      }
      FDTD_QUAD_H(1, hy, b, wz[q], a, ihx);
      // Hz
      ld4(w, en + e_pitch);
#pragma unroll
      for (int q = 0; q < 4; ++q) a[q] = w[q] - e1[q];
      ld4(w, ec + P);
#pragma unroll
      for (int q = 0; q < 4; ++q) b[q] = w[q] - e0[q];
      if (!kFold) FDTD_QUAD_SCALE(a, ihx, b, ihy);
      if (kCpml) {
        if (sxh >= 0)
          psi4<false>(a, fx, p.psiHin[2][0], p.psiHout[2][0], xslab_off(p, sxh, jc, k), fl & kValid, wr, none);
        if (wf & kYSlab)
          psi4<false>(b, fy, p.psiHin[2][1], p.psiHout[2][1], yoff(p, i, jc, k, NY - 1), fl & kYSlabH, wr, none);
      }
      FDTD_QUAD_H(2, hz, a, ihx, b, ihy);
#undef FDTD_QUAD_SCALE
#undef FDTD_QUAD_H
      if (wf & kWarpZFace) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const bool out = q >= static_cast<int>(fl & kZLast);
          hx[q] = out ? 0.f : hx[q];
          hy[q] = out ? 0.f : hy[q];
        }
      }
      if (wf & kYLast) {
        const bool ylast = fl & kYLast;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          hx[q] = ylast ? 0.f : hx[q];
          hz[q] = ylast ? 0.f : hz[q];
        }
      }
      if (i == NX - 1) {
        fill4(hy, 0.f);
        fill4(hz, 0.f);
      }
      if (tmask & terms.h_bits) quad_terms<kFold>(terms, tmask & terms.h_bits, 3, n, i, j, k, hx, hy, hz);
      // One writer for each quad of the ring: a thread that repeats the last item
      // reads the same H^{n-1/2} and, writing too, could be read by the item's own
      // thread before that has loaded it (the lanes of a warp need not run together).
      if (own && (fl & kItem)) {
        st4(hown, hx);
        st4(hown + h_pitch, hy);
        st4(hown + 2 * h_pitch, hz);
        if (fl & kOwn) {
          stcg4(p.Hout[0] + o, hx);
          stcg4(p.Hout[1] + o, hy);
          stcg4(p.Hout[2] + o, hz);
        }
      }
    }
    // the H written above lies in slots that later bulk copies overwrite
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    plane_sync();
    // ---------------- E^{n+1}(i) ----------------
    if (own && (wf & kOwn)) {
      const ZFace zf{(fl & kZFirst) != 0, static_cast<int>(fl & kZLast)};
      const ZFace none{false, 4};
      const bool yface = fl & kYFace;
      const float iex = kUniform ? p.inv_e_u[0] : __ldg(p.inv_e[0] + i);
      float wz[4], zb[4], zc[4], zik[4], a[4], b[4], w[4], v0[4], v1[4], v2[4];
      if (kUniform) fill4(wz, p.inv_e_u[2]);
      else ldg4(wz, p.ztab_e + 3 * P + k);
      Prof fx{0.f, 0.f, 1.f}, fy{0.f, 0.f, 1.f};
      if (kCpml) {
        if (sxe >= 0) fx = prof(p.eb[0], p.ec[0], p.eik[0], i);
        if ((wf & kYSlab) && (fl & kYSlabE)) fy = prof(p.eb[1], p.ec[1], p.eik[1], j);
      }
      auto scaled = [](float d, float inv) { return kFold ? d : __fmul_rn(d, inv); };
      auto curl = [&](float u, float iu, float v, float iv) { return kFold ? fold(u, iu, v, iv) : u - v; };
      // Ex: dHz/dy - dHy/dz; Ey: dHx/dz - dHz/dx; Ez: dHy/dx - dHx/dy.  psi of
      // cells that are not updated stays as it is (on a wrapped face it belongs to
      // the wrap kernel).
#define FDTD_QUAD_E(I, V, E, AB)                                                                    \
  do {                                                                                                \
    float g[4], c[4];                                                                                 \
    fill4(g, p.edecay_u[I]);                                                                          \
    fill4(c, p.ecurl_u[I]);                                                                           \
    if (kCoef && (wf & kWarpECoef)) {                                                                           \
      if (p.ecurl[I]) ldg4(c, p.ecurl[I] + o);                                                        \
      if (p.edecay[I]) ldg4(g, p.edecay[I] + o);                                                      \
    }                                                                                                 \
    _Pragma("unroll") for (int q = 0; q < 4; ++q) V[q] = __fmaf_rn(E[q], g[q], __fmul_rn(c[q], AB)); \
  } while (0)
      const float hyk = k > 0 ? hown[h_pitch - 1] : 0.f;
      ld4(w, hown + 2 * h_pitch - P);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        a[q] = scaled(hz[q] - w[q], iey);
        b[q] = scaled(hy[q] - (q > 0 ? hy[q > 0 ? q - 1 : 0] : hyk), wz[q]);
      }
      if (kCpml) {
        if (wf & kYSlab) psi4<true>(a, fy, p.psiE[0][0], p.psiE[0][0], yoff(p, i, jc, k, NY), fl & kYSlabE, true, zf);
        if (wf & kZSlab) {
          ztab(zb, zc, zik, c.ztable + 3 * p.SZ, p.SZ);
          psi4z<true>(b, zb, zc, zik, zq + 2 * c.za, p.psiE[0][1] + zslab_off(p, i, jc, k), (fl & kZSlabE) && !yface,
                      true,
                zf);
        }
      }
      FDTD_QUAD_E(0, v0, e0, curl(a[q], iey, b[q], wz[q]));
      const float hxk = k > 0 ? hown[-1] : 0.f;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        a[q] = scaled(hz[q] - hpz[q], iex);
        b[q] = scaled(hx[q] - (q > 0 ? hx[q > 0 ? q - 1 : 0] : hxk), wz[q]);
      }
      if (kCpml) {
        if (sxe >= 0) psi4<true>(a, fx, p.psiE[1][0], p.psiE[1][0], xslab_off(p, sxe, jc, k), fl & kOwn, true, zf);
        if ((wf & kZSlab) && !xface) {
          ztab(zb, zc, zik, c.ztable + 3 * p.SZ, p.SZ);
          psi4z<true>(b, zb, zc, zik, zq + 3 * c.za, p.psiE[1][1] + zslab_off(p, i, jc, k), fl & kZSlabE, true, zf);
        }
      }
      FDTD_QUAD_E(1, v1, e1, curl(b[q], wz[q], a[q], iex));
      ld4(w, hown - P);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        a[q] = scaled(hy[q] - hpy[q], iex);
        b[q] = scaled(hx[q] - w[q], iey);
      }
      if (kCpml) {
        if (sxe >= 0)
          psi4<true>(a, fx, p.psiE[2][0], p.psiE[2][0], xslab_off(p, sxe, jc, k), (fl & kOwn) && !yface, true, none);
        if ((wf & kYSlab) && !xface)
          psi4<true>(b, fy, p.psiE[2][1], p.psiE[2][1], yoff(p, i, jc, k, NY), fl & kYSlabE, true, none);
      }
      FDTD_QUAD_E(2, v2, e2, curl(a[q], iex, b[q], iey));
#undef FDTD_QUAD_E
      const bool xpec = (i == 0 && p.bnd[0] == BND_PEC) || (i == NX - 1 && p.bnd[1] == BND_PEC);
      const bool ypec = fl & kYPec;
      if (xface || (wf & kYFace)) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          if (yface) v0[q] = ypec ? 0.f : e0[q];
          if (xface) v1[q] = xpec ? 0.f : e1[q];
          if (xface || yface) v2[q] = xpec || ypec ? 0.f : e2[q];
        }
      }
      if (wf & kWarpZFace) {
        const bool zp0 = p.bnd[4] == BND_PEC, zp1 = p.bnd[5] == BND_PEC;
        if (zf.first) {
          v0[0] = zp0 || ypec ? 0.f : e0[0];
          v1[0] = zp0 || xpec ? 0.f : e1[0];
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (q == zf.last) {
            v0[q] = zp1 || ypec ? 0.f : e0[q];
            v1[q] = zp1 || xpec ? 0.f : e1[q];
          }
      }
      if (tmask & ~terms.h_bits) {
        quad_terms<kFold>(terms, tmask & ~terms.h_bits, 0, n, i, j, k, v0, v1, v2);
        // scenes without TFSF end the E update on PEC faces (stepping.py:2316-2318)
        if (p.pec_clamp) {
          const bool zp0 = zf.first && p.bnd[4] == BND_PEC, zp1 = p.bnd[5] == BND_PEC;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const bool zp = (q == 0 && zp0) || (q == zf.last && zp1);
            if (ypec || zp) v0[q] = 0.f;
            if (xpec || zp) v1[q] = 0.f;
            if (xpec || ypec) v2[q] = 0.f;
          }
        }
      }
      if (fl & kOwn) {
        stcg4(p.Eout[0] + o, v0);
        stcg4(p.Eout[1] + o, v1);
        stcg4(p.Eout[2] + o, v2);
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      hpz[q] = hz[q];
      hpy[q] = hy[q];
    }
    o += ps;
    se = sen;
    if (se == 0) par ^= 1u;
  }
}

template <bool kCpml, bool kCoef, bool kUniform>
__global__ void __launch_bounds__(quad_max_threads(kCpml), 1)
    quad_step_kernel(const __grid_constant__ StepParams p, const __grid_constant__ QuadTerms terms,
                     const QuadShape shape, int n) {
  extern __shared__ __align__(128) float smem[];
  if (p.step_base) n += __ldg(p.step_base);
  const int NX = p.NX, NY = p.NY, NZ = p.NZ, P = p.P, Q = P / 4;
  const Tile t{(static_cast<int>(blockIdx.x) + p.rb0) * shape.TY, shape.TY};
  const int chunk = static_cast<int>(blockIdx.z) + p.ch0;
  const int i0 = chunk * p.CX, i1 = min(i0 + p.CX, NX), istart = max(i0 - 1, 0);
  const int e_pitch = (shape.TY + 2) * P, h_pitch = (shape.TY + 1) * P;
  const int es = 3 * e_pitch, hs = 3 * h_pitch;  // slot sizes
  float* ering = smem;
  float* hring = smem + kSlots * es;
  float* zring = hring + kSlots * hs;               // z-slab psi: 4 arrays of TY + 1 rows
  const int zs = 4 * (shape.TY + 1) * p.SZ;
  float* ztable = zring + kSlots * zs;              // z profiles on the slab columns: H then E, b, c, 1/kappa each
  const uint32_t bar0 = saddr(ztable + 6 * p.SZ);
  for (int x = threadIdx.x; x < 6 * p.SZ; x += blockDim.x) {
    const int row = x / p.SZ, col = x - row * p.SZ;
    const int kz = col < p.zlo4 ? col : col - p.zlo4 + p.zhs4;
    ztable[x] = __ldg((row < 3 ? p.ztab_h : p.ztab_e) + (row % 3) * P + kz);
  }
  if (threadIdx.x < kSlots)
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar0 + 8u * threadIdx.x) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  __syncthreads();
  if (static_cast<int>(threadIdx.x) >= shape.threads - 32) {
    copy_march(p, t, ering, hring, zring, es, hs, zs, bar0, istart, i1, threadIdx.x & 31);
    return;
  }

  // ---- the thread's quad ----
  // Items are the quads of rows j0 - 1 .. j0 + TY - 1; the first and last few
  // quads of each row (z faces and slabs) come first, so that their code runs in
  // a few warps only.  Threads past the last item repeat it and store nothing,
  // neither to memory nor to the ring.
  const int rows = shape.TY + 1, ns = shape.nlo + shape.nhi, items = rows * Q;
  const int item = min(static_cast<int>(threadIdx.x), items - 1);
  int r, col;
  if (item < rows * ns) {
    r = item / ns;
    const int c = item - r * ns;
    col = c < shape.nlo ? c : Q - ns + c;
  } else {
    const int x = item - rows * ns, w = Q - ns;
    r = x / w;
    col = shape.nlo + x - r * w;
  }
  const int j = t.j0 - 1 + r, k = 4 * col;
  const bool valid = j >= 0 && j < NY;
  const bool eitem = valid && r >= 1 && static_cast<int>(threadIdx.x) < items;
  const int jc = min(max(j, 0), NY - 1);
  // Faces.  Cells outside a component's extent hold zero and stay zero by the
  // arithmetic alone once Hx, Hy of k >= NZ - 1, Hx, Hz of row NY - 1 and Hy, Hz
  // of plane NX - 1 are set to zero.  E on a face is kept (zeroed on PEC).
  // The flags are packed: a register each would spill.
  unsigned fl = k <= NZ - 1 && k + 4 > NZ - 1 ? NZ - 1 - k : 4;  // kZLast: cell NZ - 1 of the quad (4: not here)
  if (k == 0) fl |= kZFirst;
  if (valid) fl |= kValid;
  if (static_cast<int>(threadIdx.x) < items) fl |= kItem;
  if (eitem) fl |= kOwn;
  if (j == 0 || j == NY - 1) fl |= kYFace;
  if (j == NY - 1) fl |= kYLast;
  if ((j == 0 && p.bnd[2] == BND_PEC) || (j == NY - 1 && p.bnd[3] == BND_PEC)) fl |= kYPec;
  // Injection terms that meet the quad in some plane of the chunk
  unsigned tmask = 0;
  for (int b = 0; b < terms.n; ++b) {
    const InjectionTerm& q = terms.t[b];
    if (valid && j >= q.j0 && j < q.j1 && k + 4 > q.k0 && k < q.k1 && i1 > q.i0 && istart < q.i1 &&
        (eitem || q.comp >= 3))
      tmask |= 1u << b;
  }
  unsigned cls = 0;
  if (kCoef) cls = __ldg(p.quad_class + (static_cast<int64_t>(chunk) * NY + jc) * Q + col);
  if (kCpml && valid) {
    const bool zs = p.slab_lo[2] + p.slab_hi[2] > 0;
    if (slab_coord(p, 1, j, NY - 1) >= 0) fl |= kYSlabH;
    if (eitem && !(fl & kYFace) && slab_coord(p, 1, j, NY) >= 0) fl |= kYSlabE;
    if (zs && (k < p.slab_lo[2] || k + 3 >= NZ - 1 - p.slab_hi[2])) fl |= kZSlabH;
    if (zs && eitem && (k < p.slab_lo[2] || k + 3 >= NZ - p.slab_hi[2])) fl |= kZSlabE;
  }
  // What some lane of the warp needs: the branches on these are uniform
  unsigned wf = __reduce_or_sync(kFull, fl);
  if (__any_sync(kFull, (fl & kZFirst) || (fl & kZLast) < 4)) wf |= kWarpZFace;
  if (kCoef && __any_sync(kFull, (cls & kQuadECoef) && eitem)) wf |= kWarpECoef;
  if (kCoef && __any_sync(kFull, cls & kQuadHCoef)) wf |= kWarpHCoef;
  // x slabs make every warp of the chunk a slab warp
  bool cpml = false;
  if (kCpml) {
    cpml = (wf & (kYSlab | kZSlab)) != 0;
    const int xl = p.slab_lo[0], xh = NX - 1 - p.slab_hi[0];
    cpml = cpml || istart < xl || (p.slab_hi[0] > 0 && i1 > xh);
  }
  const int zcol = k < p.zlo4 ? k : p.zlo4 + k - p.zhs4;  // column of the quad in a z-slab psi row
  unsigned fold = 0;
  if (kCpml && slab_coord(p, 1, j, NY - 1) < 0 && slab_coord(p, 1, j, NY) < 0 && slab_coord(p, 1, j - 1, NY - 1) < 0) {
    for (int q = 0; q < 4; ++q) {
      const int b = (k + q) / kOut * kOut;
      if ((p.slab_lo[2] == 0 || b - 1 >= p.slab_lo[2]) && (p.slab_hi[2] == 0 || b + kOut < NZ - 1 - p.slab_hi[2]))
        fold |= 1u << q;
    }
  }
  const Quad q{j, k, jc, fl, wf, fold, tmask, r * P + k, istart, i0, i1, e_pitch, h_pitch, ering, hring,
               zring + r * p.SZ + zcol, ztable + zcol, zs, (shape.TY + 1) * p.SZ, bar0};
  if (kCpml && cpml) {
    if (kCoef && (wf & (kWarpECoef | kWarpHCoef))) quad_march<true, true, kUniform, false>(p, terms, q, n);
    else quad_march<true, false, kUniform, false>(p, terms, q, n);
  } else {
    if (kCoef && (wf & (kWarpECoef | kWarpHCoef))) quad_march<false, true, kUniform, !kCpml>(p, terms, q, n);
    else quad_march<false, false, kUniform, !kCpml>(p, terms, q, n);
  }
}

// One thread per (chunk, row, quad): do the E (planes [i0, i1)) or H (planes
// [istart, i1)) coefficient arrays of the quad hold a value other than the
// component's background scalar?
__global__ void quad_classify_kernel(const StepParams p, int n_chunks, unsigned char* out) {
  const int Q = p.P / 4;
  const int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= static_cast<int64_t>(n_chunks) * p.NY * Q) return;
  const int k = 4 * static_cast<int>(t % Q);
  const int j = static_cast<int>((t / Q) % p.NY);
  const int i0 = static_cast<int>(t / (static_cast<int64_t>(Q) * p.NY)) * p.CX;
  const int i1 = min(i0 + p.CX, p.NX), istart = max(i0 - 1, 0);
  unsigned bits = 0;
  for (int c = 0; c < 6; ++c) {
    const bool e = c < 3;
    const float* dec = e ? p.edecay[c] : p.hdecay[c - 3];
    const float* cur = e ? p.ecurl[c] : p.hcurl[c - 3];
    if (!dec && !cur) continue;
    const float du = e ? p.edecay_u[c] : p.hdecay_u[c - 3], cu = e ? p.ecurl_u[c] : p.hcurl_u[c - 3];
    // Yee extents: E component a ends one cell earlier along a, H along the other two
    const int ex = p.NX - ((e ? c == 0 : c != 3) ? 1 : 0), ey = p.NY - ((e ? c == 1 : c != 4) ? 1 : 0);
    const int ez = p.NZ - ((e ? c == 2 : c != 5) ? 1 : 0);
    if (j >= ey) continue;
    bool other = false;
    for (int i = e ? i0 : istart; i < min(i1, ex) && !other; ++i)
      for (int q = 0; q < 4; ++q) {
        if (k + q >= ez) break;
        const int64_t o = (static_cast<int64_t>(i) * p.NY + j) * p.P + k + q;
        other = other || (dec && __ldg(dec + o) != du) || (cur && __ldg(cur + o) != cu);
      }
    if (other) bits |= e ? kQuadECoef : kQuadHCoef;
  }
  // cells whose coefficients an instantaneous nonlinearity rewrites every step
  if (p.nl_lo[0] < p.nl_hi[0] && istart < p.nl_hi[0] && i1 > p.nl_lo[0] && j >= p.nl_lo[1] && j < p.nl_hi[1] &&
      k + 4 > p.nl_lo[2] && k < p.nl_hi[2])
    bits |= kQuadECoef;
  out[t] = static_cast<unsigned char>(bits);
}

// z tables padded to the pitch: b, c, 1/kappa of a profile, neutral outside the
// slabs, and the inverse spacing.  b == nullptr: no CPML.
__global__ void quad_ztable_kernel(const float* b, const float* c, const float* ik, const float* inv, int extent,
                                   int lo, int hi, int P, float* out) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= P) return;
  const bool in = b && k < extent && (k < lo || k >= extent - hi);
  out[k] = in ? b[k] : 0.f;
  out[P + k] = in ? c[k] : 0.f;
  out[2 * P + k] = in ? ik[k] : 1.f;
  out[3 * P + k] = k < extent ? inv[k] : 0.f;
}

}  // namespace

size_t quad_smem_bytes(int TY, int P, int SZ) {
  const size_t fields = 3 * static_cast<size_t>((TY + 2) + (TY + 1)) * P, psi = 4 * static_cast<size_t>(TY + 1) * SZ;
  return sizeof(float) * (kSlots * (fields + psi) + 6 * static_cast<size_t>(SZ)) + kSlots * sizeof(uint64_t);
}

int launch_quad_classify(const StepParams& p, int n_chunks, unsigned char* out, cudaStream_t stream) {
  const int64_t n = static_cast<int64_t>(n_chunks) * p.NY * (p.P / 4);
  quad_classify_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, stream>>>(p, n_chunks, out);
  return static_cast<int>(cudaGetLastError());
}

int launch_quad_ztable(const float* b, const float* c, const float* ik, const float* inv, int extent, int lo, int hi,
                       int P, float* out, cudaStream_t stream) {
  quad_ztable_kernel<<<(P + 127) / 128, 128, 0, stream>>>(b, c, ik, inv, extent, lo, hi, P, out);
  return static_cast<int>(cudaGetLastError());
}

namespace {
using QuadKernel = void (*)(StepParams, QuadTerms, QuadShape, int);
template <bool kCpml, bool kCoef>
QuadKernel quad_kernel_of(bool uni) {
  return uni ? quad_step_kernel<kCpml, kCoef, true> : quad_step_kernel<kCpml, kCoef, false>;
}
QuadKernel quad_kernel_of(bool cpml, bool coef, bool uni) {
  if (cpml) return coef ? quad_kernel_of<true, true>(uni) : quad_kernel_of<true, false>(uni);
  return coef ? quad_kernel_of<false, true>(uni) : quad_kernel_of<false, false>(uni);
}
}  // namespace

int prepare_quad_step(bool cpml, bool coef, bool uni) {
  return static_cast<int>(cudaFuncSetAttribute(quad_kernel_of(cpml, coef, uni),
                                               cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               static_cast<int>(kQuadMaxSmem)));
}

int launch_quad_step(const StepParams& p, const QuadTerms& terms, const QuadShape& s, int n, dim3 grid,
                     bool coef, bool uni, cudaStream_t stream) {
  const QuadKernel kern = quad_kernel_of(p.cpml != 0, coef, uni);
  kern<<<grid, s.threads, quad_smem_bytes(s.TY, p.P, p.SZ), stream>>>(p, terms, s, n);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace fdtdb200
