// Pointwise kernel of the B200 RHS + RK path.
//
//   k_thermo      pointwise: TEMPER (src/temper.f:58-219), transport
//                 properties (src/rhscal.f:515-571, 1292-1340, 3854-3885;
//                 src/rhsvel.f:933-952), species enthalpy (rhscal.f:1444-1466)
//                 and CHRATE (src/chrate.f:146-741), fused per grid point.
// The stencil kernels of the substage are in kernels_tiled.cu, the
// operator-level derivative family in deriv_ops.cu.
#include <cuda_runtime.h>

#include <cstdint>

#include <cstdlib>
#include <cstring>

#include "mech_gen.cuh"
#include "senga_internal.h"
#include "thermo.cuh"

namespace senga {

namespace {

// Resident blocks per SM asked of the compiler for a policy (register cap
// 65536 / (256 * blocks)): more warps hide the FP64 dependency chains of the
// long straight-line mechanisms.
template <class M>
struct ThermoOcc {
  static constexpr int blocks = 1;
};
#ifndef SENGA_THERMO_H2_MINB
#define SENGA_THERMO_H2_MINB 2
#endif
template <>
struct ThermoOcc<gen::Mech_h2> {
  static constexpr int blocks = SENGA_THERMO_H2_MINB;
};

template <class M>
__global__ void __launch_bounds__(kBlock, ThermoOcc<M>::blocks) k_thermo(Geo g, Fields f, M m) {
  const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= g.n) return;
  thermo_point(g, f, m, q);
}
// The two halves of the thermochemistry, each at three blocks per SM. Both
// are bound by the FP64 pipe (about 2600 and 1300 FP64 instructions a point
// when every step, pair and quotient had its own exp and divide); the
// generated forms share one exp among polynomials that differ in a constant,
// form reverse rates from one exp per species, and sum quotients as running
// fractions (gen_mech.py). 256^3 H2 box: part 1 3.76 -> 2.52, part 2 1.69 ->
// 1.17 ms per launch; 32^3: 17.3 -> 10.4 and 7.6 -> 6.2 us.
#ifndef SENGA_THERMO_P1_MINB
#define SENGA_THERMO_P1_MINB 3
#endif
#ifndef SENGA_THERMO_P2_MINB
#define SENGA_THERMO_P2_MINB 3
#endif
#ifndef SENGA_THERMO_P1_BLOCK
#define SENGA_THERMO_P1_BLOCK kBlock
#endif
#ifndef SENGA_THERMO_P2_BLOCK
#define SENGA_THERMO_P2_BLOCK kBlock
#endif
template <int PART>
constexpr int kPartBlock = PART == 1 ? SENGA_THERMO_P1_BLOCK : SENGA_THERMO_P2_BLOCK;
template <class M, int PART>
__global__ void __launch_bounds__(kPartBlock<PART>, PART == 1 ? SENGA_THERMO_P1_MINB : SENGA_THERMO_P2_MINB)
    k_thermo_part(Geo g, Fields f, M m) {
  const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= g.n) return;
  thermo_point<M, PART>(g, f, m, q);
}

// Batched: CTAs stride over (box, 256-point chunk) items.
template <class M>
__global__ void __launch_bounds__(kBlock) k_thermo_b(const __grid_constant__ BoxTable t,
                                                     const WorkItem* __restrict__ chunks, int nchunks, M m) {
  for (int it = blockIdx.x; it < nchunks; it += gridDim.x) {
    const WorkItem w = chunks[it];
    const BoxDesc& sd = t.d[w.box];
    const int64_t q = (int64_t)w.x0 * kBlock + threadIdx.x;
    if (q < sd.g.n) thermo_point(sd.g, sd.f, m, q);
  }
}

inline unsigned grid_of(int64_t n) { return (unsigned)((n + kBlock - 1) / kBlock); }

}  // namespace

int select_mech(const senga_chem& chem, const senga_diff& diff) {
  const char* env = std::getenv("SENGA_MECH");
  if (env && std::strcmp(env, "generic") == 0) return 0;
  if (gen::Mech_onestep::matches(chem, diff)) return 1;
  if (gen::Mech_h2::matches(chem, diff)) return 2;
  return 0;
}

int launch_thermo(const Geo& g, const Fields& f, const senga_chem* dchem, const senga_diff* ddiff, int nspec,
                  int flmavt, int mech, cudaStream_t s) {
  const unsigned gr = grid_of(g.n);
  if (mech == 1) {
    k_thermo<<<gr, kBlock, 0, s>>>(g, f, gen::Mech_onestep{});
  } else if (mech == 2) {
    constexpr int b1 = kPartBlock<1>, b2 = kPartBlock<2>;
    const unsigned g1 = (unsigned)((g.n + b1 - 1) / b1), g2 = (unsigned)((g.n + b2 - 1) / b2);
    if (f.err) {  // adaptive time step: see Mech_h2_ref (gen_mech.py)
      k_thermo_part<gen::Mech_h2_ref, 1><<<g1, b1, 0, s>>>(g, f, gen::Mech_h2_ref{});
      k_thermo_part<gen::Mech_h2_ref, 2><<<g2, b2, 0, s>>>(g, f, gen::Mech_h2_ref{});
    } else {
      k_thermo_part<gen::Mech_h2, 1><<<g1, b1, 0, s>>>(g, f, gen::Mech_h2{});
      k_thermo_part<gen::Mech_h2, 2><<<g2, b2, 0, s>>>(g, f, gen::Mech_h2{});
    }
    return 2;
  } else if (nspec <= 2) {
    if (flmavt) k_thermo<<<gr, kBlock, 0, s>>>(g, f, MechTables<2, true>{dchem, ddiff, nspec});
    else k_thermo<<<gr, kBlock, 0, s>>>(g, f, MechTables<2, false>{dchem, ddiff, nspec});
  } else {
    return launch_thermo_tables(g, f, dchem, ddiff, nspec, flmavt, s);
  }
  return 1;
}

cudaError_t load_thermo() {
  return load_kernels(k_thermo<gen::Mech_onestep>, k_thermo<MechTables<2, true>>, k_thermo<MechTables<2, false>>,
                      k_thermo_part<gen::Mech_h2, 1>, k_thermo_part<gen::Mech_h2, 2>,
                      k_thermo_part<gen::Mech_h2_ref, 1>, k_thermo_part<gen::Mech_h2_ref, 2>);
}

void launch_batch_thermo(const BoxTable& boxes, const WorkItem* chunks, int nchunks, int grid, int mech,
                         const senga_chem* dchem, const senga_diff* ddiff, int nspec, int flmavt, cudaStream_t s) {
  if (mech == 1) {
    k_thermo_b<<<grid, kBlock, 0, s>>>(boxes, chunks, nchunks, gen::Mech_onestep{});
  } else if (mech == 2) {
    k_thermo_b<<<grid, kBlock, 0, s>>>(boxes, chunks, nchunks, gen::Mech_h2{});
  } else if (nspec <= 2) {
    if (flmavt) k_thermo_b<<<grid, kBlock, 0, s>>>(boxes, chunks, nchunks, MechTables<2, true>{dchem, ddiff, nspec});
    else k_thermo_b<<<grid, kBlock, 0, s>>>(boxes, chunks, nchunks, MechTables<2, false>{dchem, ddiff, nspec});
  } else {
    if (flmavt) k_thermo_b<<<grid, kBlock, 0, s>>>(boxes, chunks, nchunks, MechTables<9, true>{dchem, ddiff, nspec});
    else k_thermo_b<<<grid, kBlock, 0, s>>>(boxes, chunks, nchunks, MechTables<9, false>{dchem, ddiff, nspec});
  }
}

int thermo_block() { return kBlock; }

}  // namespace senga
