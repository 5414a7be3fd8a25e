// Declarations of the quad-tile fused step kernel (quad_kernel.cu).
#pragma once

#include "engine.cuh"

namespace fdtdb200 {

// Threads of the largest CTA, and the registers that leaves each.  The slab code
// spills at 80 registers (192 x 192 x 160 with a 10-cell CPML: 136 us against 122
// with 96); without CPML 80 are enough and let 20 % more warps run.
constexpr int quad_max_threads(bool cpml) { return cpml ? 640 : 768; }
constexpr int quad_regs(bool cpml) { return cpml ? 96 : 80; }
// Longest z pitch: one row and its halo row fit a CTA.
constexpr int kQuadMaxPitch = 512;
constexpr size_t kQuadMaxSmem = 227 * 1024;

// Bits of StepParams::quad_class.
constexpr unsigned kQuadECoef = 1u;
constexpr unsigned kQuadHCoef = 2u;

// Tile of a CTA: TY owned z rows.
struct QuadShape {
  int TY;
  int nlo, nhi;  // first and last quads of a row that hold z-face or z-slab cells
  int threads;   // quads of TY + 1 rows rounded up to whole warps, and the copy warp
};

// Injection terms, read from the kernel parameters (constant bank).
constexpr int kQuadMaxTerms = 24;
struct QuadTerms {
  int n;
  unsigned h_bits;  // terms on H components
  InjectionTerm t[kQuadMaxTerms];
};

// SZ: floats of a z-slab psi row (0 without z slabs).
size_t quad_smem_bytes(int TY, int P, int SZ);
// Once per engine, on its device, before its first launch: opts the engine's kernel in
// to the largest tile's shared memory.  The limit belongs to the function and the
// device, which other engines and threads share, so it is the same for every engine:
// set to the launch's own size, it could be lowered by another thread in between.
int prepare_quad_step(bool cpml, bool coef, bool uni);
int launch_quad_step(const StepParams& p, const QuadTerms& terms, const QuadShape& s, int n, dim3 grid, bool coef,
                     bool uni, cudaStream_t stream);
// Class table [chunk][NY][P / 4] of the current chunk length p.CX.
int launch_quad_classify(const StepParams& p, int n_chunks, unsigned char* out, cudaStream_t stream);
// out: [4][P] b, c, 1/kappa (neutral outside the slabs) and inverse spacing of
// the z axis.
int launch_quad_ztable(const float* b, const float* c, const float* ik, const float* inv, int extent, int lo, int hi,
                       int P, float* out, cudaStream_t stream);

}  // namespace fdtdb200
