// sm_103a kernels of the FDTD step loop.
//
// One fused kernel per half-step replaces the reference's per-chunk dispatch
// (step_H_fused!/step_E_fused!, src/Kernels/Kernels.jl:164-454): the curl,
// the CPML cascade (Helpers.jl:30-270, CUDAKernels.jl:150-281), the
// constitutive update (Helpers.jl:323-409), source injection
// (Sources.jl:346-357) and, on the E half, the χ3 correction
// (Dispersive.jl:127-147) and the ADE pole update (Dispersive.jl:25-88) all
// happen in one pass over the grid.
//
// Work decomposition: a warp owns 32 × VN consecutive x cells of one row and
// marches over kPlanesPerCta z planes; the CTA holds kBlockY rows.  x
// neighbours come from warp shuffles, the z-neighbour plane is carried in
// registers from the previous plane (2.5D register rotation), y neighbours are
// vector loads that hit L1/L2 (the row above belongs to the next warp of the
// same CTA).
//
// Every array a thread needs for its VN cells is loaded as one vector before
// any arithmetic, so a plane costs one memory round trip also in CPML rows.
//
// Which arrays a cell touches is a static property of the cell:
//  * plain cells (no CPML region flag, no source/χ3/pole) keep no B/D state:
//    O += m⁻¹·K.  This equals m⁻¹·(T + K) of the reference up to rounding and
//    is exact when m⁻¹ = 1;
//  * all other cells keep B/D and follow the reference's stage logic for the
//    CPML auxiliaries their region allocates (Chunking.jl:1069-1146).
#include <cuda_runtime.h>

#include <algorithm>

#include "kh_cell.cuh"
#include "kh_lean.cuh"

namespace kh {

#ifdef KH_DEBUG_BOUNDS
KH_DBG_READER(dbg_read_kernels)
#endif

template <typename T, int VN>
struct PlaneLoads {
  T l0[VN], l1[VN], a2[VN], y0[VN], y2[VN];  // A0/A1 fresh plane, A2, y neighbours
  T xn1, xn2;                                // x neighbours of A1/A2 for the edge lanes
  T O[3][VN], m[3][VN];
  T t[3][VN], u[3][VN], w[3][VN], c3[VN];
  uint32_t cls[VN];
  bool tf;                                   // plane's tile holds special cells
};

template <typename T, int VN, bool H, bool FULL>
__device__ __forceinline__ void load_plane(const HalfStepParams<T>& p, PlaneLoads<T, VN>& L, int k,
                                           long long row, int lane, bool row_end, bool lane_ok, bool pervox,
                                           bool fy, bool anyfx, uint64_t tbits) {
  constexpr int s = H ? 1 : -1;
  const long long q = row + (long long)k * p.plane;
  vzero(L.l0); vzero(L.l1); vzero(L.a2); vzero(L.y0); vzero(L.y2);
  L.xn1 = T(0);
  L.xn2 = T(0);
  L.tf = ((tbits >> (k & 63)) & 1ull) != 0;
  const bool fz = k < p.pml_lo[2] || k >= p.nz - p.pml_hi[2];
  const bool anyRegion = fy || fz || anyfx;
  const bool axis_any[3] = {anyfx, fy, fz};
  if (lane_ok) {
    if constexpr (H) {  // l = A(k+1)
      vld_at(p.A[0], q + p.plane, p.total, 3001, L.l0);
      vld_at(p.A[1], q + p.plane, p.total, 3001, L.l1);
    } else {  // l = A(k)
      vld_at(p.A[0], q, p.total, 3001, L.l0);
      vld_at(p.A[1], q, p.total, 3001, L.l1);
    }
    vld_at(p.A[2], q, p.total, 3002, L.a2);
    vld_at(p.A[0], q + s * p.pitch, p.total, 3003, L.y0);
    vld_at(p.A[2], q + s * p.pitch, p.total, 3003, L.y2);
    if constexpr (H) {
      if (row_end && KH_IN(q + VN, p.total, 3004)) {
        L.xn1 = p.A[1][q + VN];
        L.xn2 = p.A[2][q + VN];
      }
    } else {
      if (lane == 0 && KH_IN(q - 1, p.total, 3004)) {
        L.xn1 = p.A[1][q - 1];
        L.xn2 = p.A[2][q - 1];
      }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) vld_at(p.O[c], q, p.total, 3005, L.O[c]);
    if (pervox) {
#pragma unroll
      for (int c = 0; c < 3; ++c) vld_at(p.m_inv[c], q, p.total, 3006, L.m[c]);
    }
#pragma unroll
    for (int v = 0; v < VN; ++v)
      L.cls[v] = (L.tf && lane_ok && KH_IN(q + v, p.total, 3007)) ? p.cell_class[q + v] : 0u;
    const bool aux = anyRegion || L.tf;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      if (aux && p.Ts[c]) vld_at(p.Ts[c], q, p.total, 3008, L.t[c]); else vzero(L.t[c]);
      if (anyRegion && p.U[c] && axis_any[(c + 1) % 3]) vld_at(p.U[c], q, p.total, 3009, L.u[c]);
      else vzero(L.u[c]);
      if (anyRegion && p.W[c] && axis_any[c]) vld_at(p.W[c], q, p.total, 3010, L.w[c]); else vzero(L.w[c]);
    }
    if (FULL && !H && L.tf && p.chi3) vld_at(p.chi3, q, p.total, 3011, L.c3); else vzero(L.c3);
  } else {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      vzero(L.O[c]); vzero(L.t[c]); vzero(L.u[c]); vzero(L.w[c]);
    }
    vzero(L.c3);
#pragma unroll
    for (int v = 0; v < VN; ++v) L.cls[v] = 0u;
  }
  if (!pervox) {
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int v = 0; v < VN; ++v) L.m[c][v] = p.m_scalar;
  }
}

// Update of plane k from its loads L; r0/r1 carry the rotated z-neighbour
// plane of A0/A1 in and out.
template <typename T, int VN, bool H, bool CPML, bool FULL>
__device__ __forceinline__ void compute_plane(const HalfStepParams<T>& p, PlaneLoads<T, VN>& L, int k,
                                              long long row, int lane, bool row_end, bool lane_ok, int x0,
                                              int j, bool fy, bool anyfx, const bool (&fxv)[VN],
                                              const AxisCoef<T> (&axv)[VN], const AxisCoef<T>& ay,
                                              T (&r0)[VN], T (&r1)[VN]) {
  const long long q = row + (long long)k * p.plane;
  // cur = A0/A1 at plane k, nb = at plane k+s
  const T(&cur0)[VN] = H ? r0 : L.l0;
  const T(&cur1)[VN] = H ? r1 : L.l1;
  const T(&nb0)[VN] = H ? L.l0 : r0;
  const T(&nb1)[VN] = H ? L.l1 : r1;

  // x neighbours of A1 and A2 at plane k
  T x1s[VN], x2s[VN];
  if constexpr (H) {
    T n1 = __shfl_down_sync(0xffffffffu, cur1[0], 1);
    T n2 = __shfl_down_sync(0xffffffffu, L.a2[0], 1);
    if (row_end) {
      n1 = L.xn1;
      n2 = L.xn2;
    }
#pragma unroll
    for (int v = 0; v < VN - 1; ++v) { x1s[v] = cur1[v + 1]; x2s[v] = L.a2[v + 1]; }
    x1s[VN - 1] = n1;
    x2s[VN - 1] = n2;
  } else {
    T n1 = __shfl_up_sync(0xffffffffu, cur1[VN - 1], 1);
    T n2 = __shfl_up_sync(0xffffffffu, L.a2[VN - 1], 1);
    if (lane == 0) {
      n1 = L.xn1;
      n2 = L.xn2;
    }
#pragma unroll
    for (int v = 1; v < VN; ++v) { x1s[v] = cur1[v - 1]; x2s[v] = L.a2[v - 1]; }
    x1s[0] = n1;
    x2s[0] = n2;
  }

  if (lane_ok) {
    T K[3][VN];
#pragma unroll
    for (int v = 0; v < VN; ++v) {
      K[0][v] = p.dt * (p.inv_d[2] * (nb1[v] - cur1[v]) - p.inv_d[1] * (L.y2[v] - L.a2[v]));
      K[1][v] = p.dt * (p.inv_d[0] * (x2s[v] - L.a2[v]) - p.inv_d[2] * (nb0[v] - cur0[v]));
      K[2][v] = p.dt * (p.inv_d[1] * (L.y0[v] - cur0[v]) - p.inv_d[0] * (x1s[v] - cur1[v]));
    }
    const bool fz = k < p.pml_lo[2] || k >= p.nz - p.pml_hi[2];
    const bool anyRegion = fy || fz || anyfx;
    bool anySpecial = false;
#pragma unroll
    for (int v = 0; v < VN; ++v) anySpecial |= (L.cls[v] & (H ? kSpecialH : kSpecialE)) != 0;
    if (!anyRegion && !anySpecial) {
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int v = 0; v < VN; ++v) L.O[c][v] = L.O[c][v] + L.m[c][v] * K[c][v];
    } else {
      const AxisCoef<T> az = KH_IN(k, p.nz, 3012) ? p.ax[2][k] : AxisCoef<T>{T(0), T(1), T(1), T(1)};
#pragma unroll
      for (int v = 0; v < VN; ++v) {
        const int i = x0 + v;
        if (i >= p.nx) continue;
        const bool special = (L.cls[v] & (H ? kSpecialH : kSpecialE)) != 0;
        if (!(fxv[v] || fy || fz || special)) {
#pragma unroll
          for (int c = 0; c < 3; ++c) L.O[c][v] = L.O[c][v] + L.m[c][v] * K[c][v];
          continue;
        }
        const bool fc[3] = {fxv[v], fy, fz};
        const AxisCoef<T> ac[3] = {axv[v], ay, az};
        const T Kc[3] = {K[0][v], K[1][v], K[2][v]};
        const T mc[3] = {L.m[0][v], L.m[1][v], L.m[2][v]};
        T Oc[3] = {L.O[0][v], L.O[1][v], L.O[2][v]};
        T tc[3] = {L.t[0][v], L.t[1][v], L.t[2][v]};
        T uc[3] = {L.u[0][v], L.u[1][v], L.u[2][v]};
        T wc[3] = {L.w[0][v], L.w[1][v], L.w[2][v]};
        if constexpr (FULL) {
          general_cell<T, H>(p, q + v, i, j, k, fc, ac, L.cls[v], special, Kc, mc, Oc, tc, uc, wc, L.c3[v]);
        } else {
          if (fc[0] || fc[1] || fc[2]) {
            pml_cell<T, CPML>(fc, ac, Kc, mc, Oc, tc, uc, wc);
          } else {  // source cell outside CPML: keeps its B|D state
#pragma unroll
            for (int c = 0; c < 3; ++c) {
              tc[c] = tc[c] + Kc[c];
              Oc[c] = mc[c] * tc[c];
            }
          }
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          L.O[c][v] = Oc[c];
          L.t[c][v] = tc[c];
          L.u[c][v] = uc[c];
          L.w[c][v] = wc[c];
        }
      }
      const bool axis_any[3] = {anyfx, fy, fz};
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        if (p.Ts[c]) vst_at(p.Ts[c], q, p.total, 3013, L.t[c]);
        if (p.U[c] && axis_any[(c + 1) % 3]) vst_at(p.U[c], q, p.total, 3014, L.u[c]);
        if (p.W[c] && axis_any[c]) vst_at(p.W[c], q, p.total, 3015, L.w[c]);
      }
    }
    if (x0 + VN <= p.nx) {
#pragma unroll
      for (int c = 0; c < 3; ++c) vst_at(p.O[c], q, p.total, 3016, L.O[c]);
    } else {
#pragma unroll
      for (int v = 0; v < VN; ++v) {
        if (x0 + v < p.nx && KH_IN(q + v, p.total, 3017)) {
#pragma unroll
          for (int c = 0; c < 3; ++c) p.O[c][q + v] = L.O[c][v];
        }
      }
    }
  }
  // rotate: H half keeps A(k+1) as the next plane's A(k); E half keeps
  // A(k) as the next plane's A(k-1)
#pragma unroll
  for (int v = 0; v < VN; ++v) { r0[v] = L.l0[v]; r1[v] = L.l1[v]; }
}

// One fused half-step.  H = true: B/H from curl E; H = false: D/E from curl H.
// FULL = false (LEAN) compiles only plain and CPML cells; cells marked special
// there are source cells, updated as B|D-keeping cells (O = m⁻¹·T) and given
// their source term by source_fix_kernel when sources are active.
//
// The z march is double-buffered with a prefetch distance of two planes: the
// loads of plane k+2 are issued as soon as plane k has been consumed, so each
// warp keeps about two planes of memory traffic in flight.
template <typename T, int VN, bool H, bool CPML, bool FULL>
__global__ void __launch_bounds__(32 * kBlockY, sizeof(T) == 4 ? kMinBlocks : 2)
    half_step_kernel(const HalfStepParams<T> p) {
  const int lane = threadIdx.x;
  const int j = blockIdx.y * kBlockY + threadIdx.y;
  if (j >= p.ny) return;  // warp-uniform: blockDim.x == 32
  const int xb = blockIdx.x;
  const int x0 = (xb * 32 + lane) * VN;
  const bool lane_ok = x0 < p.nx;
  // nobody in the warp has this lane's right neighbour: at the row's end that is the
  // ring, the face across where x is periodic
  const bool row_end = lane == 31 || x0 + VN >= p.nx;
  const int k0 = blockIdx.z * kPlanesPerCta;
  const int k1 = min(k0 + kPlanesPerCta, p.nz);
  const long long row = p.origin + (long long)j * p.pitch + x0;
  const bool fy = j < p.pml_lo[1] || j >= p.ny - p.pml_hi[1];
  const bool pervox = p.m_inv[0] != nullptr;
  // special-tile bits of planes [64·(k0/64), +64) of this warp's row segment
  const long long tbi = ((long long)(k0 >> 6) * p.ny + j) * p.nxb + xb;
  const uint64_t tbits = (p.tile_bits && KH_IN(tbi, p.n_tile_words, 3018)) ? p.tile_bits[tbi] : 0ull;

  // per-cell x flags and CPML coefficients of this thread's vector and the
  // row's y coefficients: static along the z march
  bool fxv[VN];
  AxisCoef<T> axv[VN];
  bool anyfx = false;
#pragma unroll
  for (int v = 0; v < VN; ++v) {
    const int i = x0 + v;
    fxv[v] = i < p.nx && (i < p.pml_lo[0] || i >= p.nx - p.pml_hi[0]);
    anyfx |= fxv[v];
    axv[v] = (i < p.nx && KH_IN(i, p.nx, 3019)) ? p.ax[0][i] : AxisCoef<T>{T(0), T(1), T(1), T(1)};
  }
  const AxisCoef<T> ay = KH_IN(j, p.ny, 3020) ? p.ax[1][j] : AxisCoef<T>{T(0), T(1), T(1), T(1)};

  // rotated z-neighbour plane of A0, A1: A(k0) for the H half, A(k0-1) for E
  T r0[VN], r1[VN];
  vzero(r0);
  vzero(r1);
  if (lane_ok) {
    const long long q0 = row + (long long)k0 * p.plane + (H ? 0 : -p.plane);
    vld_at(p.A[0], q0, p.total, 3021, r0);
    vld_at(p.A[1], q0, p.total, 3021, r1);
  }
  PlaneLoads<T, VN> A, B;
  load_plane<T, VN, H, FULL>(p, A, k0, row, lane, row_end, lane_ok, pervox, fy, anyfx, tbits);
  if (k0 + 1 < k1) load_plane<T, VN, H, FULL>(p, B, k0 + 1, row, lane, row_end, lane_ok, pervox, fy, anyfx, tbits);
  for (int k = k0; k < k1; k += 2) {
    compute_plane<T, VN, H, CPML, FULL>(p, A, k, row, lane, row_end, lane_ok, x0, j, fy, anyfx, fxv, axv, ay, r0, r1);
    if (k + 2 < k1) load_plane<T, VN, H, FULL>(p, A, k + 2, row, lane, row_end, lane_ok, pervox, fy, anyfx, tbits);
    if (k + 1 < k1) {
      compute_plane<T, VN, H, CPML, FULL>(p, B, k + 1, row, lane, row_end, lane_ok, x0, j, fy, anyfx, fxv, axv, ay, r0, r1);
      if (k + 3 < k1) load_plane<T, VN, H, FULL>(p, B, k + 3, row, lane, row_end, lane_ok, pervox, fy, anyfx, tbits);
    }
  }
}

template <typename T, bool CPML, bool FULL>
static void launch_variant(bool h_half, const HalfStepParams<T>& p, cudaStream_t st) {
  dim3 block(32, kBlockY, 1);
  dim3 grid(p.nxb, (p.ny + kBlockY - 1) / kBlockY, (p.nz + kPlanesPerCta - 1) / kPlanesPerCta);
  if (h_half) half_step_kernel<T, kVN, true, CPML, FULL><<<grid, block, 0, st>>>(p);
  else half_step_kernel<T, kVN, false, CPML, FULL><<<grid, block, 0, st>>>(p);
}

template <typename T>
void launch_half_step(bool h_half, const HalfStepParams<T>& p, void* stream) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (p.cpml) {
    if (p.full) launch_variant<T, true, true>(h_half, p, st);
    else launch_variant<T, true, false>(h_half, p, st);
  } else {
    if (p.full) launch_variant<T, false, true>(h_half, p, st);
    else launch_variant<T, false, false>(h_half, p, st);
  }
}

// Source term of the cells a LEAN half-step updated as B|D-keeping cells:
// O = m⁻¹·(T + S), the same arithmetic update_field_generic performs
// (net = T; net += S; A = m⁻¹·net, Helpers.jl:329-347).
// Component c of source cell q: O = m⁻¹·(T + S), or through the W stage
// when the cell lies in the CPML of c's own axis (SourceFixParams).
template <typename T>
__device__ __forceinline__ T source_fix_cell(const SourceFixParams<T>& p, long long q, int c, T S) {
  const T m = p.m_inv[c] ? p.m_inv[c][q] : p.m_scalar;
  T net = p.Ts[c][q];
  net += S;
  if (p.W[c]) {
    const long long rel = q - p.origin;
    int idx;
    if (p.total <= 0xffffffffll) {  // 32-bit division wherever the offsets fit
      const unsigned r = unsigned(rel), plane = unsigned(p.plane), pitch = unsigned(p.pitch);
      const unsigned k = r / plane, rem = r - k * plane, j = rem / pitch;
      idx = int(c == 0 ? rem - j * pitch : (c == 1 ? j : k));
    } else {
      const long long k = rel / p.plane, rem = rel % p.plane;
      idx = c == 0 ? int(rem % p.pitch) : (c == 1 ? int(rem / p.pitch) : int(k));
    }
    if ((idx < p.pml_lo[c] || idx >= p.n[c] - p.pml_hi[c]) && KH_IN(idx, p.n[c], 3031)) {
      const AxisCoef<T> ao = p.ax[c][idx];
      if (ao.s != T(0)) {
        const T wl = p.W[c][q];
        const T wn = m * net;
        p.W[c][q] = wn;
        const T o = p.O[c][q] + ao.op * (wn - wl);
        p.O[c][q] = o;
        return o;
      }
    }
  }
  const T o = m * net;
  p.O[c][q] = o;
  return o;
}

template <typename T>
__device__ __forceinline__ void source_fix_one(const SourceFixParams<T>& p, long long q, int c, T S) {
  const T o = source_fix_cell(p, q, c, S);
  if (!p.wrap) return;
  // the ghost copies that the half-step made of a face cell
  const long long rel = q - p.origin;
  const int k = int(rel / p.plane);
  const long long rem = rel - (long long)k * p.plane;
  const int j = int(rem / p.pitch);
  const int at[3] = {int(rem - (long long)j * p.pitch), j, k};
  const long long st[3] = {1, p.pitch, p.plane};
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    if (!((p.wrap >> a) & 1u)) continue;
    const long long d = (long long)p.n[a] * st[a];
    if (at[a] == 0 && KH_IN(q + d, p.total, 3032)) p.O[c][q + d] = o;
    if (at[a] == p.n[a] - 1 && KH_IN(q - d, p.total, 3033)) p.O[c][q - d] = o;
  }
}

template <typename T>
__global__ void source_fix_kernel(const SourceFixParams<T> p) {
  const int slot = blockIdx.x * blockDim.x + threadIdx.x;
  if (slot >= p.nslots) return;
  const long long q = p.slot_cell[slot];
  const SlotPack<T> pk = p.slot_pack[slot];
  if (!KH_IN(q, p.total, 3022)) return;
  const int base = p.h_half ? 3 : 0;
  if (pk.src >= 0) {  // a single entry: one component, S = real(f(t)·amplitude)
    const int c = pk.comp - base;
    if (c < 0 || c > 2 || !KH_IN(pk.src, p.n_src, 3024)) return;
    const Cplx<T> f = p.f_now[pk.src];
    T S = T(0);
    S += f.re * pk.amp.re - f.im * pk.amp.im;
    source_fix_one(p, q, c, S);
    return;
  }
  T S[3] = {T(0), T(0), T(0)};
  bool has[3] = {false, false, false};
  for (int e = p.slot_off[slot]; e < p.slot_off[slot + 1]; ++e) {
    if (!KH_IN(e, p.n_ent, 3023)) break;
    const int c = p.ent_comp[e] - base;
    if (c < 0 || c > 2) continue;
    const Cplx<T> a = p.ent_amp[e];
    if (!KH_IN(p.ent_src[e], p.n_src, 3024)) continue;
    const Cplx<T> f = p.f_now[p.ent_src[e]];
    const T v = f.re * a.re - f.im * a.im;
    if (c == 0) { S[0] += v; has[0] = true; }
    else if (c == 1) { S[1] += v; has[1] = true; }
    else { S[2] += v; has[2] = true; }
  }
#pragma unroll
  for (int c = 0; c < 3; ++c)
    if (has[c]) source_fix_one(p, q, c, S[c]);
}

template <typename T>
void launch_source_fix(const SourceFixParams<T>& p, void* stream) {
  if (p.nslots <= 0) return;
  const int threads = 128;
  source_fix_kernel<T><<<(p.nslots + threads - 1) / threads, threads, 0, static_cast<cudaStream_t>(stream)>>>(p);
}

// ---------------------------------------------------------------------------
// Dispersive and Kerr cells after a LEAN E half-step (DispFixParams).  One
// warp per entry of the row-segment list (32·kVN cells).  A segment without
// pole cells needs no class words: its lanes load the pair of E vectors and
// χ3 values of their two cells at once and correct the cells with χ3 ≠ 0
// (the cells the LEAN launch left uncorrected).  Pole segments go through the
// class words, pair by pair (256³ with a χ3 slab and two poles' spheres: 57 to 52 µs
// a launch against cell by cell; reading σ first to leave out absent poles puts
// a round trip before the rest: 58).
template <typename T>
__global__ void disp_fix_kernel(const DispFixParams<T> p) {
  static_assert(kVN == 2, "paired loads of the χ3 path");
  const long long w = (long long)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
  if (w >= p.n_list) return;  // warp-uniform
  const uint32_t ent = p.list[w];
  const unsigned seg = ent & 0x7fffffffu;
  const unsigned r = seg / unsigned(p.nxb);
  const int xb = int(seg - r * unsigned(p.nxb));
  const int k = int(r / unsigned(p.ny));
  const int j = int(r - unsigned(k) * unsigned(p.ny));
  const int lane = threadIdx.x & 31;
  const int i0 = xb * 32 * kVN + lane * kVN;
  const long long q0 = p.origin + (long long)k * p.plane + (long long)j * p.pitch + i0;
  if (!(ent >> 31)) {
    if (!p.chi3 || i0 >= p.nx) return;
    if (i0 + 1 < p.nx && KH_IN(q0 + 1, p.total, 3045)) {
      using V2 = typename VT<T, 2>::V;  // q0 is even: 8/16-byte aligned
      // the E pair is loaded with the χ3 pair (one round trip, not two):
      // in a Kerr segment nearly every cell has χ3
      const V2 c3 = *reinterpret_cast<const V2*>(p.chi3 + q0);
      V2 e[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) e[c] = *reinterpret_cast<const V2*>(p.E[c] + q0);
      if (c3.x == T(0) && c3.y == T(0)) return;
      // χ3 Kerr correction (Dispersive.jl:127-147), same operation order as below
      if (c3.x != T(0)) {
        const T esq = (e[0].x * e[0].x + e[1].x * e[1].x) + e[2].x * e[2].x;
        const T corr = T(1) / (T(1) + c3.x * esq);
#pragma unroll
        for (int c = 0; c < 3; ++c) e[c].x = e[c].x * corr;
      }
      if (c3.y != T(0)) {
        const T esq = (e[0].y * e[0].y + e[1].y * e[1].y) + e[2].y * e[2].y;
        const T corr = T(1) / (T(1) + c3.y * esq);
#pragma unroll
        for (int c = 0; c < 3; ++c) e[c].y = e[c].y * corr;
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) *reinterpret_cast<V2*>(p.E[c] + q0) = e[c];
      return;
    }
  }
  // Both cells of a lane at once: every array is read as a pair (the row padding
  // makes the second one readable past an odd row's end), so a lane's loads of a
  // stage are in flight together.
  if (i0 >= p.nx || !(KH_IN(q0, p.total, 3040) && KH_IN(q0 + 1, p.total, 3040))) return;
  using V2 = typename VT<T, 2>::V;
  const bool two = i0 + 1 < p.nx;
  const uint2 cl = *reinterpret_cast<const uint2*>(p.cell_class + q0);
  const uint32_t cls[2] = {cl.x, two ? cl.y : 0u};
  if (!((cls[0] | cls[1]) & (kHasChi3 | kHasPole))) return;
  auto ld = [&](const T* a, T (&x)[2]) {
    const V2 w = *reinterpret_cast<const V2*>(a + q0);
    x[0] = w.x;
    x[1] = w.y;
  };
  auto st = [&](T* a, const T (&x)[2]) {
    if (two) {
      V2 w;
      w.x = x[0];
      w.y = x[1];
      *reinterpret_cast<V2*>(a + q0) = w;
    } else {
      a[q0] = x[0];
    }
  };
  const bool pole[2] = {(cls[0] & kHasPole) != 0, (cls[1] & kHasPole) != 0};
  T O[3][2], c3[2] = {T(0), T(0)};
#pragma unroll
  for (int c = 0; c < 3; ++c) ld(p.E[c], O[c]);
  if (p.chi3) ld(p.chi3, c3);
  if (pole[0] || pole[1]) {
    T D[3][2], m[3][2], Ptot[3][2] = {};
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      ld(p.D[c], D[c]);
      if (p.m_inv[c]) ld(p.m_inv[c], m[c]);
      else m[c][0] = m[c][1] = p.m_scalar;
    }
    for (int pp = 0; pp < p.npoles; ++pp) {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        T P[2];
        ld(p.poles[pp].P[c], P);
        Ptot[c][0] += P[0];
        Ptot[c][1] += P[1];
      }
    }
#pragma unroll
    for (int v = 0; v < 2; ++v) {
      if (!pole[v]) continue;
      // E = ε⁻¹·(D + S − Σ P) (update_field_generic: net = T; net += S; net -= P)
      T S[3] = {T(0), T(0), T(0)};
      bool hasS[3] = {false, false, false};
      if (p.sources_active && (cls[v] & kHasSrcE)) {
        const int slot = int(cls[v] >> kSlotShift);
        if (KH_IN(slot + 1, p.n_slots + 1, 3041)) {
          for (int e = p.slot_off[slot]; e < p.slot_off[slot + 1]; ++e) {
            if (!KH_IN(e, p.n_ent, 3042) || !KH_IN(p.ent_src[e], p.n_src, 3043)) continue;
            const int c = p.ent_comp[e];
            const Cplx<T> am = p.ent_amp[e];
            const Cplx<T> fv = p.f_now[p.ent_src[e]];
            const T x = fv.re * am.re - fv.im * am.im;  // real(f(t) · amplitude)
#pragma unroll
            for (int o = 0; o < 3; ++o)
              if (c == o) {
                S[o] += x;
                hasS[o] = true;
              }
          }
        }
      }
      const int i = i0 + v;
      const long long q = q0 + v;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        T net = D[c][v];
        if (hasS[c]) net += S[c];
        net -= Ptot[c][v];
        const T e0 = O[c][v];
        O[c][v] = m[c][v] * net;
        // in the CPML of its own axis the cell's E comes out of the W stage
        // (update_field_generic, Helpers.jl:333-339): E = E' + op·(W_new − W')
        // on top of the W' and E' that the LEAN launch (or the source kernel)
        // left, W_new = ε⁻¹·net
        if (p.W[c]) {
          const int idx = c == 0 ? i : (c == 1 ? j : k);
          const int nn = c == 0 ? p.nx : (c == 1 ? p.ny : p.nz);
          if ((idx < p.pml_lo[c] || idx >= nn - p.pml_hi[c]) && KH_IN(idx, nn, 3046)) {
            const AxisCoef<T> ao = p.ax[c][idx];
            if (ao.s != T(0)) {
              const T wl = p.W[c][q];
              const T wn = m[c][v] * net;
              p.W[c][q] = wn;
              O[c][v] = e0 + ao.op * (wn - wl);
            }
          }
        }
      }
    }
  }
#pragma unroll
  for (int v = 0; v < 2; ++v) {
    // χ3 Kerr correction (Dispersive.jl:127-147)
    if ((cls[v] & kHasChi3) && c3[v] != T(0)) {
      const T esq = (O[0][v] * O[0][v] + O[1][v] * O[1][v]) + O[2][v] * O[2][v];
      const T corr = T(1) / (T(1) + c3[v] * esq);
#pragma unroll
      for (int c = 0; c < 3; ++c) O[c][v] = O[c][v] * corr;
    }
  }
  // ADE poles with E^{n+1} (Dispersive.jl:25-88)
  if (pole[0] || pole[1]) {
    for (int pp = 0; pp < p.npoles; ++pp) {
      const PoleParams<T>& P = p.poles[pp];
      T s[2], px[3][2], pv[3][2];
      ld(P.sigma, s);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        ld(P.P[c], px[c]);
        ld(P.Pprev[c], pv[c]);
      }
      const bool act[2] = {pole[0] && s[0] != T(0), pole[1] && s[1] != T(0)};
      if (!(act[0] || act[1])) continue;
      const T cp = P.is_drude ? T(2) : P.coeff_p;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
#pragma unroll
        for (int v = 0; v < 2; ++v) {
          if (!act[v]) continue;
          const T pn = P.gamma1_inv * ((cp * px[c][v] - P.gamma1 * pv[c][v]) + (P.drive * s[v]) * O[c][v]);
          pv[c][v] = px[c][v];
          px[c][v] = pn;
        }
        st(P.P[c], px[c]);
        st(P.Pprev[c], pv[c]);
      }
    }
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) st(p.E[c], O[c]);
}

template <typename T>
void launch_disp_fix(const DispFixParams<T>& p, void* stream) {
  if (p.n_list <= 0) return;
  const int warps = 8;
  disp_fix_kernel<T><<<unsigned((p.n_list + warps - 1) / warps), 32 * warps, 0,
                       static_cast<cudaStream_t>(stream)>>>(p);
}

// ---------------------------------------------------------------------------
// Periodic wrap after a half-step of the general or the register-pipelined kernel
// (the reduced-state one writes its ghost layers itself).  One block row per periodic axis and component:
// blockIdx.y = 3·(index of the axis in p.axes) + component; threads stride
// over the face's (n_t1 × n_t2) cells, t1 the lower of the face's two axes;
// each copies both directions of one cell.
template <typename T>
__global__ void wrap_kernel(const WrapParams<T> p) {
  const int a = p.axes[blockIdx.y / 3], c = blockIdx.y % 3;
  // the face's lower axis runs fastest across threads: x on the y and z
  // faces (coalesced rows), y on the x face (one element per row there)
  const int t1 = a == 0 ? 1 : 0, t2 = a == 2 ? 1 : 2;
  const long long st[3] = {1, p.pitch, p.plane};
  const long long face = (long long)p.n[t1] * p.n[t2];
  T* f = p.O[c];
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < face;
       e += (long long)gridDim.x * blockDim.x) {
    long long u, v;
    if (face <= 0xffffffffll) {  // 32-bit division wherever the face fits
      const unsigned w = unsigned(e) / unsigned(p.n[t1]);
      v = w;
      u = unsigned(e) - w * unsigned(p.n[t1]);
    } else {
      u = e % p.n[t1];
      v = e / p.n[t1];
    }
    const long long base = p.origin + u * st[t1] + v * st[t2];
    const long long lo = base, hi = base + (long long)(p.n[a] - 1) * st[a];
    const long long ghost_lo = base - st[a], ghost_hi = base + (long long)p.n[a] * st[a];
    if (!(KH_IN(ghost_lo, p.total, 3028) && KH_IN(ghost_hi, p.total, 3029))) continue;
    const T fh = f[hi], fl = f[lo];  // both on their way before the first store
    if (!(p.chi3 && p.chi3[hi] != T(0))) f[ghost_lo] = fh;
    if (!(p.chi3 && p.chi3[lo] != T(0))) f[ghost_hi] = fl;
  }
}

template <typename T>
void launch_wrap(const WrapParams<T>& p0, void* stream) {
  if (!(p0.periodic & 7u)) return;
  WrapParams<T> p = p0;
  int na = 0;
  long long face = 0;
  for (int a = 0; a < 3; ++a)
    if ((p.periodic >> a) & 1u) {
      p.axes[na++] = a;
      face = std::max(face, (long long)p.n[(a + 1) % 3] * p.n[(a + 2) % 3]);
    }
  const int threads = 256;
  const long long blocks = std::min<long long>((face + threads - 1) / threads, 1024);
  wrap_kernel<T><<<dim3(unsigned(std::max<long long>(blocks, 1)), unsigned(3 * na)), threads, 0,
                   static_cast<cudaStream_t>(stream)>>>(p);
}

// ---------------------------------------------------------------------------
// DFT accumulation (update_dft_monitor!, Monitors.jl:361-379):
//   F[cell, f] += Δt·exp(i2πf t)·field[cell]
// FP32 accumulators carry a Kahan compensation term.  One update, shared by
// the per-monitor and the batched kernels so both give the same bits.
template <typename T>
__device__ __forceinline__ void dft_add(Cplx<T>& acc, Cplx<T>& c, Cplx<T> ph, T v) {
  const T yr = fma_rn(ph.re, v, -c.re);
  const T yi = fma_rn(ph.im, v, -c.im);
  const T tr = add_rn(acc.re, yr);
  const T ti = add_rn(acc.im, yi);
  c.re = sub_rn(sub_rn(tr, acc.re), yr);
  c.im = sub_rn(sub_rn(ti, acc.im), yi);
  acc.re = tr;
  acc.im = ti;
}

template <typename T>
__device__ __forceinline__ void dft_add(Cplx<T>& acc, Cplx<T> ph, T v) {
  acc.re = fma_rn(ph.re, v, acc.re);
  acc.im = fma_rn(ph.im, v, acc.im);
}

template <typename T>
__device__ __forceinline__ void dft_update(Cplx<T>* F, Cplx<T>* comp, long long t, Cplx<T> ph, T v) {
  Cplx<T> acc = F[t];
  if (comp) {
    Cplx<T> c = comp[t];
    dft_add(acc, c, ph, v);
    comp[t] = c;
  } else {
    dft_add(acc, ph, v);
  }
  F[t] = acc;
}

template <typename T>
__global__ void dft_kernel(const DftParams<T> p) {
  const long long ncell = (long long)p.dims[0] * p.dims[1] * p.dims[2];
  const long long total = ncell * p.nf;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const int f = int(t / ncell);
    const long long cell = t - (long long)f * ncell;
    const int i = int(cell % p.dims[0]);
    const long long r = cell / p.dims[0];
    const int jj = int(r % p.dims[1]);
    const int kk = int(r / p.dims[1]);
    const long long q = p.origin + (long long)(p.start[2] + kk) * p.plane +
                        (long long)(p.start[1] + jj) * p.pitch + (p.start[0] + i);
    if (!KH_IN(q, p.total, 3025)) continue;
    dft_update(p.F, p.comp, t, p.phase[f], p.field[q]);
  }
}

// kDftThreads·VEC cells and up to p.freqs frequencies of one monitor.  A thread
// finds its VEC consecutive cells and reads the field once, then goes through the
// frequencies with the accumulators of four of them in flight.
template <typename T, int VEC>
__device__ __forceinline__ void dft_block(const DftBatchParams<T>& p, const typename DftBatchParams<T>::Mon& M,
                                          unsigned u, long long ncell) {
  struct alignas(sizeof(Cplx<T>) * VEC) Acc {
    Cplx<T> v[VEC];
  };
  const unsigned groups = unsigned(M.nf + p.freqs - 1) / unsigned(p.freqs);
  const long long cell = ((long long)(u / groups) * kDftThreads + threadIdx.x) * VEC;
  if (cell >= ncell) return;
  const int f0 = int(u % groups) * p.freqs, f1 = min(f0 + p.freqs, M.nf);
  T x[VEC];
#pragma unroll
  for (int e = 0; e < VEC; ++e) {
    // 32-bit division wherever the cell index fits
    const unsigned row = ncell <= 0xffffffffll ? unsigned(cell + e) / unsigned(M.dims[0])
                                               : unsigned((cell + e) / M.dims[0]);
    const int i = int(cell + e - (long long)row * M.dims[0]);
    const int kk = int(row / unsigned(M.dims[1])), jj = int(row % unsigned(M.dims[1]));
    const long long q = p.origin + (long long)(M.start[2] + kk) * p.plane + (long long)(M.start[1] + jj) * p.pitch +
                        (M.start[0] + i);
    if (!KH_IN(q, p.total, 3030)) return;
    x[e] = M.field[q];
  }
  const bool kahan = M.comp != nullptr;
  char* F = reinterpret_cast<char*>(M.F + (long long)f0 * ncell + cell);
  char* C = kahan ? reinterpret_cast<char*>(M.comp + (long long)f0 * ncell + cell) : nullptr;
  const long long step = ncell * (long long)sizeof(Cplx<T>);
  constexpr int kFly = 4;
  for (int f = f0; f < f1; f += kFly) {
    Acc a[kFly], c[kFly];
#pragma unroll
    for (int w = 0; w < kFly; ++w)
      if (f + w < f1) {
        a[w] = *reinterpret_cast<const Acc*>(F + w * step);
        if (kahan) c[w] = *reinterpret_cast<const Acc*>(C + w * step);
      }
#pragma unroll
    for (int w = 0; w < kFly; ++w)
      if (f + w < f1) {
        const Cplx<T> ph = M.phase[f + w];
#pragma unroll
        for (int e = 0; e < VEC; ++e) {
          if (kahan) dft_add(a[w].v[e], c[w].v[e], ph, x[e]);
          else dft_add(a[w].v[e], ph, x[e]);
        }
        *reinterpret_cast<Acc*>(F + w * step) = a[w];
        if (kahan) *reinterpret_cast<Acc*>(C + w * step) = c[w];
      }
    F += kFly * step;
    if (kahan) C += kFly * step;
  }
}

// Cells per thread of the batched kernel: 16 bytes of accumulators, unless the
// launch is small (freqs = 1).  A monitor with an odd number of cells takes one,
// as its frequencies' rows then start on 8 bytes.
template <typename T>
__host__ __device__ constexpr int dft_vec(long long ncell, int freqs) {
  return sizeof(T) == 4 && freqs > 1 && ncell % 2 == 0 ? 2 : 1;
}

// All monitors of one half-step in one grid: block u with first[m] <= u <
// first[m+1] belongs to monitor m.  Bound by the accumulators' traffic (32 bytes
// per cell and frequency in FP32).
template <typename T>
__global__ void __launch_bounds__(kDftThreads) dft_batch_kernel(const DftBatchParams<T> p) {
  int m = 0;
  while (m + 1 < p.n && blockIdx.x >= p.first[m + 1]) ++m;
  const auto& M = p.mon[m];
  const long long ncell = (long long)M.dims[0] * M.dims[1] * M.dims[2];
  const unsigned u = blockIdx.x - p.first[m];
  if constexpr (sizeof(T) == 4) {
    if (dft_vec<T>(ncell, p.freqs) == 2) {
      dft_block<T, 2>(p, M, u, ncell);
      return;
    }
  }
  dft_block<T, 1>(p, M, u, ncell);
}

// One item per thread while the launch is no more than the GPU holds at once
// (its time is then one chain of loads: 64³ with 3 × 1764-cell monitors 3.59
// against 3.65 ms for 256 steps); 8 frequencies × 2 cells above (256×256×128, 21
// frequencies on two planes: 42 to 24 µs a launch).
template <typename T>
void launch_dft_batch(const DftBatchParams<T>& p0, void* stream) {
  DftBatchParams<T> p = p0;
  long long items = 0;
  for (int m = 0; m < p.n; ++m)
    items += (long long)p.mon[m].dims[0] * p.mon[m].dims[1] * p.mon[m].dims[2] * p.mon[m].nf;
  if (items <= 0) return;
  p.freqs = items <= 152LL * 2048 ? 1 : kDftFreqs;
  p.first[0] = 0;
  for (int m = 0; m < p.n; ++m) {
    const long long ncell = (long long)p.mon[m].dims[0] * p.mon[m].dims[1] * p.mon[m].dims[2];
    const long long cells = (long long)kDftThreads * dft_vec<T>(ncell, p.freqs);
    p.first[m + 1] = p.first[m] + unsigned((ncell + cells - 1) / cells * ((p.mon[m].nf + p.freqs - 1) / p.freqs));
  }
  dft_batch_kernel<T><<<p.first[p.n], kDftThreads, 0, static_cast<cudaStream_t>(stream)>>>(p);
}

template <typename T>
void launch_dft(const DftParams<T>& p, void* stream) {
  const long long total = (long long)p.dims[0] * p.dims[1] * p.dims[2] * p.nf;
  int blocks = int((total + 255) / 256);
  if (blocks > 152 * 16) blocks = 152 * 16;
  if (blocks < 1) blocks = 1;
  dft_kernel<T><<<blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(p);
}

// ---------------------------------------------------------------------------
// History recording: a block row of threads per x row of a box, rows laid out x
// fastest in the destination slot; blockIdx.z is the monitor.  A few microseconds of
// launch against well under one of copying, so the three components of a design
// region go together (200×200×64 with 60×60×11 cells, two runs of 128 steps: 22.9 to 20.8 ms).
template <typename T>
__global__ void record_kernel(const RecordParams<T> p) {
  const auto& R = p.rec[blockIdx.z];
  const int rows = R.dims[1] * R.dims[2];
  for (int r = blockIdx.y * blockDim.y + threadIdx.y; r < rows; r += gridDim.y * blockDim.y) {
    const int jj = r % R.dims[1], kk = r / R.dims[1];
    const T* src = R.field + p.origin + (long long)(R.start[2] + kk) * p.plane +
                   (long long)(R.start[1] + jj) * p.pitch + R.start[0];
    T* dst = R.dst + (long long)r * R.dims[0];
    const long long s0 = src - R.field;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < R.dims[0]; i += gridDim.x * blockDim.x)
      if (KH_IN(s0 + i, p.total, 3026) &&
          KH_IN((long long)r * R.dims[0] + i, (long long)rows * R.dims[0], 3027))
        dst[i] = src[i];
  }
}

template <typename T>
void launch_record(const RecordParams<T>& p, void* stream) {
  int d0 = 1, rows = 1;
  for (int q = 0; q < p.n; ++q) {
    d0 = std::max(d0, p.rec[q].dims[0]);
    rows = std::max(rows, p.rec[q].dims[1] * p.rec[q].dims[2]);
  }
  const dim3 block(32, 4);
  const dim3 grid(unsigned(std::min((d0 + 31) / 32, 64)), unsigned(std::min((rows + 3) / 4, 65535)), unsigned(p.n));
  record_kernel<T><<<grid, block, 0, static_cast<cudaStream_t>(stream)>>>(p);
}

// ---------------------------------------------------------------------------
// Flux (get_flux, FluxMonitor.jl:92-156) in FP64: one block per frequency,
// fixed-order tree reduction so the result is reproducible.
template <typename T>
__device__ __forceinline__ void load_c(const Cplx<T>* F, const Cplx<T>* C, long long q, double& re,
                                       double& im) {
  re = double(F[q].re);
  im = double(F[q].im);
  if (C) {  // Kahan: sum - compensation
    re -= double(C[q].re);
    im -= double(C[q].im);
  }
}

struct FluxArgs {
  int d[4][3];
  int normal;
  int nf;
  double dA;
};

template <typename T>
__device__ __forceinline__ void avg_at(const Cplx<T>* F, const Cplx<T>* C, const int* d, int normal,
                                       int a1, int a2, int i1, int i2, int f, double& re,
                                       double& im) {
  int idx[3];
  idx[normal] = 0;
  idx[a1] = i1;
  idx[a2] = i2;
  const long long ncell = (long long)d[0] * d[1] * d[2];
  long long q = (long long)f * ncell + ((long long)idx[2] * d[1] + idx[1]) * d[0] + idx[0];
  load_c(F, C, q, re, im);
  if (d[normal] >= 2) {  // _avg_dim: (layer 1 + layer 2) / 2
    idx[normal] = 1;
    long long q2 = (long long)f * ncell + ((long long)idx[2] * d[1] + idx[1]) * d[0] + idx[0];
    double r2, i2v;
    load_c(F, C, q2, r2, i2v);
    re = (re + r2) / 2;
    im = (im + i2v) / 2;
  }
}

constexpr int kFluxCellsPerBlock = 1024;

template <typename T>
__global__ void flux_partial_kernel(const Cplx<T>* e1, const Cplx<T>* e2, const Cplx<T>* h1,
                                    const Cplx<T>* h2, const Cplx<T>* ce1, const Cplx<T>* ce2,
                                    const Cplx<T>* ch1, const Cplx<T>* ch2, const FluxArgs a,
                                    double* partial) {
  const int f = blockIdx.y;
  const int n = a.normal;
  const int a1 = n == 0 ? 1 : 0;
  const int a2 = n == 2 ? 1 : 2;
  int n1 = a.d[0][a1], n2 = a.d[0][a2];
  for (int m = 1; m < 4; ++m) {
    n1 = min(n1, a.d[m][a1]);
    n2 = min(n2, a.d[m][a2]);
  }
  const long long cells = (long long)n1 * n2;
  // block b takes cells [b·span, (b+1)·span), span a multiple of blockDim
  const long long span = ((cells + gridDim.x - 1) / gridDim.x + blockDim.x - 1) / blockDim.x * blockDim.x;
  const long long t0 = (long long)blockIdx.x * span;
  const long long t1 = t0 + span < cells ? t0 + span : cells;
  double acc = 0.0;
  for (long long t = t0 + threadIdx.x; t < t1; t += blockDim.x) {
    const int i1 = int(t % n1), i2 = int(t / n1);
    double E1r, E1i, E2r, E2i, H1r, H1i, H2r, H2i;
    avg_at(e1, ce1, a.d[0], n, a1, a2, i1, i2, f, E1r, E1i);
    avg_at(e2, ce2, a.d[1], n, a1, a2, i1, i2, f, E2r, E2i);
    avg_at(h1, ch1, a.d[2], n, a1, a2, i1, i2, f, H1r, H1i);
    avg_at(h2, ch2, a.d[3], n, a1, a2, i1, i2, f, H2r, H2i);
    // Re(E1·conj(H2) − E2·conj(H1))
    acc += ((E1r * H2r + E1i * H2i) - (E2r * H1r + E2i * H1i)) * a.dA;
  }
  __shared__ double red[256];
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[(long long)f * gridDim.x + blockIdx.x] = red[0];
}

// One warp per frequency: lane l adds partials l, l+32, … in order, then a
// fixed shuffle tree.
__global__ void flux_final_kernel(const double* partial, int nb, double* out) {
  const int f = blockIdx.x;
  const int lane = threadIdx.x;
  double s = 0.0;
  for (int b = lane; b < nb; b += 32) s += partial[(long long)f * nb + b];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane == 0) out[f] = s;
}

int flux_blocks(long long cells, int nf, int partial_cap) {
  long long b = (cells + kFluxCellsPerBlock - 1) / kFluxCellsPerBlock;
  const long long fill = (4LL * 152 + nf - 1) / (nf > 0 ? nf : 1);  // about four blocks per SM in all
  if (b > fill) b = fill;
  if (nf > 0 && b > partial_cap / nf) b = partial_cap / nf;
  return int(b < 1 ? 1 : b);
}

template <typename T>
void launch_flux(const Cplx<T>* e1, const Cplx<T>* e2, const Cplx<T>* h1, const Cplx<T>* h2,
                 const Cplx<T>* c_e1, const Cplx<T>* c_e2, const Cplx<T>* c_h1,
                 const Cplx<T>* c_h2, const int dims_e1[3], const int dims_e2[3],
                 const int dims_h1[3], const int dims_h2[3], int normal_axis, int nf, double dA,
                 double* out, double* partial, int partial_cap, void* stream) {
  FluxArgs a;
  for (int q = 0; q < 3; ++q) {
    a.d[0][q] = dims_e1[q];
    a.d[1][q] = dims_e2[q];
    a.d[2][q] = dims_h1[q];
    a.d[3][q] = dims_h2[q];
  }
  a.normal = normal_axis;
  a.nf = nf;
  a.dA = dA;
  if (nf <= 0) return;
  const int na1 = normal_axis == 0 ? 1 : 0, na2 = normal_axis == 2 ? 1 : 2;
  long long n1 = dims_e1[na1], n2 = dims_e1[na2];
  for (const int* d : {dims_e2, dims_h1, dims_h2}) {
    n1 = std::min<long long>(n1, d[na1]);
    n2 = std::min<long long>(n2, d[na2]);
  }
  const int nb = flux_blocks(n1 * n2, nf, partial_cap);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  flux_partial_kernel<T><<<dim3(unsigned(nb), unsigned(nf)), 256, 0, st>>>(e1, e2, h1, h2, c_e1, c_e2, c_h1,
                                                                          c_h2, a, partial);
  flux_final_kernel<<<unsigned(nf), 32, 0, st>>>(partial, nb, out);
}

template void launch_half_step<float>(bool, const HalfStepParams<float>&, void*);
template void launch_half_step<double>(bool, const HalfStepParams<double>&, void*);
template void launch_wrap<float>(const WrapParams<float>&, void*);
template void launch_wrap<double>(const WrapParams<double>&, void*);
template void launch_source_fix<float>(const SourceFixParams<float>&, void*);
template void launch_source_fix<double>(const SourceFixParams<double>&, void*);
template void launch_record<float>(const RecordParams<float>&, void*);
template void launch_record<double>(const RecordParams<double>&, void*);
template void launch_dft<float>(const DftParams<float>&, void*);
template void launch_dft_batch<float>(const DftBatchParams<float>&, void*);
template void launch_disp_fix<float>(const DispFixParams<float>&, void*);
template void launch_disp_fix<double>(const DispFixParams<double>&, void*);
template void launch_dft_batch<double>(const DftBatchParams<double>&, void*);
template void launch_dft<double>(const DftParams<double>&, void*);
template void launch_flux<float>(const Cplx<float>*, const Cplx<float>*, const Cplx<float>*,
                                 const Cplx<float>*, const Cplx<float>*, const Cplx<float>*,
                                 const Cplx<float>*, const Cplx<float>*, const int*, const int*,
                                 const int*, const int*, int, int, double, double*, double*, int, void*);
template void launch_flux<double>(const Cplx<double>*, const Cplx<double>*, const Cplx<double>*,
                                  const Cplx<double>*, const Cplx<double>*, const Cplx<double>*,
                                  const Cplx<double>*, const Cplx<double>*, const int*, const int*,
                                  const int*, const int*, int, int, double, double*, double*, int, void*);

}  // namespace kh
