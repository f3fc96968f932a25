// Launchers of the face, lifting and time-step kernels, the volume-flux dispatcher and the volume
// kernel's launch shapes.
#include <atomic>

#include "kernels.cuh"
#include "launch.h"
#include "vol_shapes.h"

namespace fluxo {

cudaError_t launch_volume_shape(int NP, int VF, bool visc, int shape, int nElems, cudaStream_t s,
                                const KParams& P) {
  switch (VF) {
    case 0: return launch_volume_vf0(NP, visc, shape, nElems, s, P);
    case 1: return launch_volume_vf1(NP, visc, shape, nElems, s, P);
    case 2: return launch_volume_vf2(NP, visc, shape, nElems, s, P);
    case 3: return launch_volume_vf3(NP, visc, shape, nElems, s, P);
    case 4: return launch_volume_vf4(NP, visc, shape, nElems, s, P);
    case 5: return launch_volume_vf5(NP, visc, shape, nElems, s, P);
    case 6: return launch_volume_vf6(NP, visc, shape, nElems, s, P);
    case 7: return launch_volume_vf7(NP, visc, shape, nElems, s, P);
    case 8: return launch_volume_vf8(NP, visc, shape, nElems, s, P);
    case 9: return launch_volume_vf9(NP, visc, shape, nElems, s, P);
    case 10: return launch_volume_vf10(NP, visc, shape, nElems, s, P);
    case 32: return launch_volume_vf32(NP, visc, shape, nElems, s, P);
    default: return cudaErrorInvalidValue;
  }
}

namespace {
// per (NP, VF, visc), shape + 1: the pinned one (0: none, the rule decides) and that of the last launch (for
// reports only)
std::atomic<int> g_pinned[10][33][2], g_used[10][33][2];

bool shape_key(int NP, int VF) { return NP >= 2 && NP <= 9 && VF >= 0 && VF <= 32; }
}  // namespace

int volume_shape_count(int NP) { return vol_shape_count(NP); }

int volume_shape(int NP, int VF, bool visc) {
  if (!shape_key(NP, VF)) return -1;
  const int pin = g_pinned[NP][VF][visc].load();
  return (pin ? pin : g_used[NP][VF][visc].load()) - 1;
}

bool pin_volume_shape(int NP, int VF, bool visc, int shape) {
  if (!shape_key(NP, VF) || shape >= vol_shape_count(NP)) return false;
  g_pinned[NP][VF][visc].store(shape < 0 ? 0 : shape + 1);
  if (shape < 0) g_used[NP][VF][visc].store(0);
  return true;
}

cudaError_t launch_volume(int NP, int VF, bool visc, int rule, int nElems, cudaStream_t s, const KParams& P) {
  if (!shape_key(NP, VF)) return cudaErrorInvalidValue;
  const int pin = g_pinned[NP][VF][visc].load(), shape = pin ? pin - 1 : rule;
  g_used[NP][VF][visc].store(shape + 1);
  return launch_volume_shape(NP, VF, visc, shape, nElems, s, P);
}

bool volume_flux_supported(int VF) {
  return (VF >= 0 && VF <= 10) || VF == 32;
}

bool riemann_supported(int RS) {
  switch (RS) {
    case 0: case 1: case 2: case 3: case 4: case 5: case 6: case 7: case 8: case 9: case 10: case 11: case 12:
    case 13: case 14: case 15: case 16: case 17: case 18: case 19: case 20: case 21: case 22: case 23: case 24:
    case 32: case 33: case 44:
      return true;
    default:
      return false;
  }
}

template <int RS, bool VISC>
static cudaError_t face_t(int NP, int nSides, cudaStream_t s, const KParams& P) {
  const int npts = NP * NP;
  const int spb = (128 / npts) > 0 ? (128 / npts) : 1;
  const int grid = (nSides + spb - 1) / spb;
  // 8 resident blocks of 128 threads per SM (64 registers): the face pass is DRAM-latency bound, and
  // the extra warps in flight outweigh the spills of the heavier Riemann solvers (measured at N=7 with
  // the matrix-dissipation solver: 4.2 TB/s against 3.5 TB/s at the unbounded 114 registers)
  return launch_k(P.pdl, face_flux_kernel<RS, VISC, 8>, grid, spb * npts, 0, s, P, NP);
}

cudaError_t launch_face_flux(int RS, bool visc, int NP, int nSides, cudaStream_t s, const KParams& P) {
#define FLUXO_RS_CASE(K) \
  case K: return visc ? face_t<K, true>(NP, nSides, s, P) : face_t<K, false>(NP, nSides, s, P);
  switch (RS) {
    FLUXO_RS_CASE(0) FLUXO_RS_CASE(1) FLUXO_RS_CASE(2) FLUXO_RS_CASE(3) FLUXO_RS_CASE(4) FLUXO_RS_CASE(5)
    FLUXO_RS_CASE(6) FLUXO_RS_CASE(7) FLUXO_RS_CASE(8) FLUXO_RS_CASE(9) FLUXO_RS_CASE(10) FLUXO_RS_CASE(11)
    FLUXO_RS_CASE(12) FLUXO_RS_CASE(13) FLUXO_RS_CASE(14) FLUXO_RS_CASE(15) FLUXO_RS_CASE(16) FLUXO_RS_CASE(17)
    FLUXO_RS_CASE(18) FLUXO_RS_CASE(19) FLUXO_RS_CASE(20) FLUXO_RS_CASE(21) FLUXO_RS_CASE(22) FLUXO_RS_CASE(23)
    FLUXO_RS_CASE(24) FLUXO_RS_CASE(32) FLUXO_RS_CASE(33) FLUXO_RS_CASE(44)
    default: return cudaErrorInvalidValue;
  }
#undef FLUXO_RS_CASE
}

cudaError_t launch_lift_flux(int NP, int nSides, cudaStream_t s, const KParams& P) {
  const size_t n = (size_t)nSides * NP * NP;
  const int grid = (int)((n + 255) / 256);
  return launch_k(P.pdl, lift_flux_kernel, grid, 256, 0, s, P, NP, P.lflux);
}

cudaError_t launch_gradient(int NP, int nElems, cudaStream_t s, const KParams& P) {
  return launch_lift_visc(NP, P.lifting, P.lifting_var, nElems, s, P);
}

template <int NP, bool VISC>
static cudaError_t dt_t(int nElems, cudaStream_t s, const KParams& P, unsigned long long* dtBits, int* errKey) {
  constexpr int NP3 = NP * NP * NP;
  constexpr int EPB = (256 / NP3) > 0 ? (256 / NP3) : 1;
  return launch_k(P.pdl, timestep_kernel<NP, VISC>, (nElems + EPB - 1) / EPB, EPB * NP3, 0, s, P, dtBits, errKey);
}

cudaError_t launch_timestep(int NP, bool visc, int nElems, cudaStream_t s, const KParams& P,
                            unsigned long long* dtBits, int* errKey) {
#define FLUXO_DT_CASE(K) \
  case K: return visc ? dt_t<K, true>(nElems, s, P, dtBits, errKey) : dt_t<K, false>(nElems, s, P, dtBits, errKey);
  switch (NP) {
    FLUXO_DT_CASE(2) FLUXO_DT_CASE(3) FLUXO_DT_CASE(4) FLUXO_DT_CASE(5)
    FLUXO_DT_CASE(6) FLUXO_DT_CASE(7) FLUXO_DT_CASE(8) FLUXO_DT_CASE(9)
    default: return cudaErrorInvalidValue;
  }
#undef FLUXO_DT_CASE
}

}  // namespace fluxo
