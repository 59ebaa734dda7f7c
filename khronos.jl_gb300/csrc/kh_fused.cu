// Whole-step kernel for sm_103a: the H and the E half of one time step in one
// pass over a grid without CPML.
//
// Two half-step launches read E twice and H twice; one pass reads E, H and ε⁻¹
// once and writes E and H once (12 instead of 18 words per cell and step with a
// uniform ε).  The new H of the low x, y and z neighbours, which E needs, is
// computed again by the tile that reads it, from the same old values, so nothing
// is waited for across CTAs; that takes the new fields into a second set of
// arrays (a neighbour may still read the old ones), and two steps bring them back.
//
// A CTA owns up to 60 × 7 cells and marches up its z chunk.  Its 8 warps hold
// one row of 64 cells each: the halo row below the tile, then the 7 rows.  Per
// plane a thread updates H of its 2 cells, passes it on (y neighbours through
// shared memory, x neighbours by shuffle, z in registers) and updates E of them.
// Planes of E (with an x/y halo on the high side), H and ε⁻¹ arrive by TMA in a
// ring of kFusedStages.  The arithmetic is that of the half-step kernel, bit for
// bit.
//
// Bound by memory and the work on the halo (8/7 of the rows, 64/32 to 64/60 of
// the columns for H).  µs a step of 216×200×168 against half-steps: dipole 106 to 71
// with a uniform ε (4.9 TB/s on 12 words a cell), 117 to 85 with per-voxel ε; a current
// plane, which flags a segment of every row, 122 to 90 and 132 to 101.  Over 138 closed
// boxes (20 to 400 cells an axis) half-steps were faster on few, all 60 to 64 cells
// wide (two half-empty column tiles): 62×150×150 30.4 against 27.5, 64×128×128 24.7
// against 23.6, 64×300×300 90 against 109.
//
// Every mbarrier wait is bounded, as in kh_lean.cu.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "../../include/khronos_gb300.h"
#include "kh_async.cuh"
#include "kh_lean.cuh"

namespace kh {

#ifdef KH_DEBUG_BOUNDS
KH_DBG_READER(dbg_read_fused)
#endif

namespace {

template <typename T, bool PV>
struct FusedGeom {
  static constexpr int HX = 16 / int(sizeof(T));  // x halo of the boxes (16 bytes)
  static constexpr int XO = xoff<T>();
  static constexpr int EX = kTmaX + HX;           // E box row length
  static constexpr int E_BYTES = EX * (kFusedRows + 1) * int(sizeof(T));
  static constexpr int E_ELEMS = ((E_BYTES + 127) / 128 * 128) / int(sizeof(T));
  static constexpr int H_ELEMS = kTmaX * kFusedRows;
  static constexpr int M_ELEMS = kTmaX * (kFusedRows - 1);
  static constexpr int STAGE = 3 * (E_ELEMS + H_ELEMS + (PV ? M_ELEMS : 0));
  static constexpr size_t SMEM = size_t(kFusedStages) * STAGE * sizeof(T) + kFusedStages * sizeof(uint64_t);
};

}  // namespace

template <typename T, bool PV, bool STALL = false>
__global__ void __launch_bounds__(32 * kFusedRows, PV ? kFusedMinBlocks : kFusedMinBlocks + 1)
    step_fused_kernel(const __grid_constant__ FusedParams<T> p, const __grid_constant__ FusedMaps maps) {
  using G = FusedGeom<T, PV>;
  constexpr int VN = 2;
  using PK = Pack<T, VN>;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  T* stages = reinterpret_cast<T*>(smem_raw);
  uint64_t* bars = reinterpret_cast<uint64_t*>(stages + kFusedStages * G::STAGE);

  const int lane = threadIdx.x;
  const int wy = threadIdx.y;
  const bool issuer = lane == 0 && wy == 0;
  const int x_own = blockIdx.x * p.tile_w;       // first owned cell
  const int x_end = min(x_own + p.tile_w, p.nx);  // past the last one
  const int X0 = x_own - G::HX;                  // first cell of the boxes
  const int y_own = blockIdx.y * (kFusedRows - 1);
  const int j = y_own - 1 + wy;
  const int x0 = X0 + lane * VN;
  const int k0 = blockIdx.z * p.zplanes;
  const int k1 = min(k0 + p.zplanes, p.nz);
  const int N = k1 - k0;
  // cells whose H this thread updates (own ones and the low halo), and own cells
  const bool row_in = j >= 0 && j < p.ny;
  const bool h_ok = row_in && x0 >= 0 && x0 + VN > x_own - 1 && x0 < x_end;
  const bool own = row_in && wy > 0 && x0 >= x_own && x0 < x_end;
  const bool full = x0 + 1 < p.nx;

  if (issuer) {
    for (int st = 0; st < kFusedStages; ++st) mbar_init(&bars[st], 1);
    mbar_fence_init();
  }
  __syncthreads();

  constexpr int kLimit = STALL ? kStallSleepWaitLimit : kSleepWaitLimit;
  const int l0 = k0 == 0 ? 1 : 0;  // nothing is updated below the grid
  // load l: plane k0 - 1 + l; the last one (plane k1) brings only what the H
  // update below it reads
  auto issue = [&](int l, int st) {
    T* dst = stages + st * G::STAGE;
    if (STALL && l == l0) {
      // failure-detection test instantiation: the first stage expects 16 bytes
      // and no copy is issued into it, so the wait on it runs out
      mbar_arrive_expect_tx(&bars[st], 16u);
      return;
    }
    const bool last = l == N + 1;
    mbar_arrive_expect_tx(&bars[st], (last ? 2u : 3u) * uint32_t(G::E_BYTES) +
                                         (last ? 0u : 3u * uint32_t(G::H_ELEMS * sizeof(T))) +
                                         (PV && !last ? 3u * uint32_t(G::M_ELEMS * sizeof(T)) : 0u));
    const int px = G::XO + X0, zc = k0 + l;  // padded coordinates
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      if (c < 2 || !last) tma_load_3d(dst + c * G::E_ELEMS, &maps.e[c], px, y_own, zc, &bars[st]);
      if (last) continue;
      tma_load_3d(dst + 3 * G::E_ELEMS + c * G::H_ELEMS, &maps.h[c], px, y_own, zc, &bars[st]);
      if constexpr (PV)
        tma_load_3d(dst + 3 * (G::E_ELEMS + G::H_ELEMS) + c * G::M_ELEMS, &maps.m[c], px, y_own + 1, zc, &bars[st]);
    }
  };
  if (issuer)
    for (int l = l0; l < min(l0 + kFusedStages, N + 2); ++l) issue(l, l - l0);

  long long q = p.origin + (long long)(k0 - 1 + l0) * p.plane + (long long)j * p.pitch + x0;
  auto put3 = [&](T* const (&arr)[3], const Cells<T, VN>& x, int site) {
    if (full) {
      if (KH_IN(q, p.total, site) && KH_IN(q + VN - 1, p.total, site)) {
#pragma unroll
        for (int c = 0; c < 3; ++c) *reinterpret_cast<PK*>(arr[c] + q) = x.c[c];
      }
    } else if (KH_IN(q, p.total, site)) {
#pragma unroll
      for (int c = 0; c < 3; ++c) arr[c][q] = x.c[c].v[0];
    }
  };
  // special-cell plane bits of this thread's 64-cell row segment, one word per
  // 64 planes; the current plane's bit is the lowest
  const long long tb_group = (long long)p.ny * p.nxb;
  auto tile_word = [&](int k) -> uint64_t {
    const long long w = (long long)j * p.nxb + (x0 >> 6) + (k >> 6) * tb_group;
    return (p.tile_bits && own && KH_IN(w, p.n_tile_words, 2203)) ? p.tile_bits[w] >> (k & 63) : 0ull;
  };
  uint64_t tbits = tile_word(k0);

  const T cd0 = p.cd[0], cd1 = p.cd[1], cd2 = p.cd[2], mu = p.mu_scalar;
  const int ea = wy * G::EX + lane * VN;  // this thread's cells in the E box
  const int ha = wy * kTmaX + lane * VN;  // … in the H box
  PK hz0{}, hz1{};                        // new H0, H1 of the plane below
  if (own && k0 == 0) {                   // … the ring below the grid
    const long long qb = q - p.plane;
    if (KH_IN(qb, p.total, 2204) && KH_IN(qb + VN - 1, p.total, 2204)) {
      hz0 = *reinterpret_cast<const PK*>(p.Ho[0] + qb);
      hz1 = *reinterpret_cast<const PK*>(p.Ho[1] + qb);
    }
  }
  int gave_up = -1;
  int st = 0;
  uint32_t parity = 0;
  if (!mbar_wait_sleep(smem_u32(bars), 0u, kLimit)) {
    gave_up = l0;
    if (p.err) atomicExch(p.err, KH_ERR_TIMEOUT);
  }
  for (int l = l0; l <= N; ++l) {
    const int sn = st + 1 == kFusedStages ? 0 : st + 1;
    const uint32_t pn = sn == 0 ? parity ^ 1u : parity;
    // special rows: class words and D on their way together, before the wait and the
    // H update, instead of one after the other between the plane's two barriers
    const bool tf = own && l > 0 && (tbits & 1ull);
    uint2 cls{0u, 0u};
    Cells<T, VN> D;
    if (tf && KH_IN(q, p.total, 2227) && KH_IN(q + VN - 1, p.total, 2227)) {
      cls = *reinterpret_cast<const uint2*>(p.cell_class + q);
#pragma unroll
      for (int c = 0; c < 3; ++c) D.c[c] = *reinterpret_cast<const PK*>(p.D[c] + q);
    }
    if (gave_up < 0 && !mbar_wait_sleep(smem_u32(bars + sn), pn, kLimit)) {
      gave_up = l;
      if (p.err) atomicExch(p.err, KH_ERR_TIMEOUT);
    }
    const bool smem_ok = KH_IN(ea + G::EX + VN, G::E_ELEMS, 2211) && KH_IN(ha + VN - 1, G::H_ELEMS, 2212);
    T* S = stages + st * G::STAGE;
    auto lds = [](const T* a) { return *reinterpret_cast<const PK*>(a); };
    const bool run = gave_up < 0 && smem_ok;
    Cells<T, VN> E{}, H{};
    if (run) {
      const T* E0 = S + ea;
      const T* E1 = E0 + G::E_ELEMS;
      const T* E2 = E1 + G::E_ELEMS;
      const T* En = stages + sn * G::STAGE + ea;
      E.c[0] = lds(E0);
      E.c[1] = lds(E1);
      E.c[2] = lds(E2);
#pragma unroll
      for (int c = 0; c < 3; ++c) H.c[c] = lds(S + 3 * G::E_ELEMS + c * G::H_ELEMS + ha);
      if (h_ok) {
        const PK y0 = lds(E0 + G::EX), y2 = lds(E2 + G::EX), n0 = lds(En), n1 = lds(En + G::E_ELEMS);
        const T e1 = E1[VN], e2 = E2[VN];
#pragma unroll
        for (int v = 0; v < VN; ++v) {
          const T x1 = v + 1 < VN ? E.c[1].v[(v + 1) % VN] : e1;
          const T x2 = v + 1 < VN ? E.c[2].v[(v + 1) % VN] : e2;
          const T k0_ = curl_rn(cd2, n1.v[v], E.c[1].v[v], cd1, y2.v[v], E.c[2].v[v]);
          const T k1_ = curl_rn(cd0, x2, E.c[2].v[v], cd2, n0.v[v], E.c[0].v[v]);
          const T k2_ = curl_rn(cd1, y0.v[v], E.c[0].v[v], cd0, x1, E.c[1].v[v]);
          H.c[0].v[v] = fma_rn(mu, k0_, H.c[0].v[v]);
          H.c[1].v[v] = fma_rn(mu, k1_, H.c[1].v[v]);
          H.c[2].v[v] = fma_rn(mu, k2_, H.c[2].v[v]);
        }
        // the y neighbour of the row above; nobody else reads the old values
        *reinterpret_cast<PK*>(S + 3 * G::E_ELEMS + ha) = H.c[0];
        *reinterpret_cast<PK*>(S + 3 * G::E_ELEMS + 2 * G::H_ELEMS + ha) = H.c[2];
        if (own && l > 0) put3(p.Hn, H, 2219);
      }
    }
    const T x1 = __shfl_up_sync(0xffffffffu, H.c[1].v[VN - 1], 1);
    const T x2 = __shfl_up_sync(0xffffffffu, H.c[2].v[VN - 1], 1);
    __syncthreads();
    if (run && own && l > 0) {
      const T* Hs = S + 3 * G::E_ELEMS + ha - kTmaX;
      const PK y0 = lds(Hs), y2 = lds(Hs + 2 * G::H_ELEMS);
      Cells<T, VN> K, m;
#pragma unroll
      for (int v = 0; v < VN; ++v) {
        const T xa = v > 0 ? H.c[1].v[(v + VN - 1) % VN] : x1;
        const T xb = v > 0 ? H.c[2].v[(v + VN - 1) % VN] : x2;
        K.c[0].v[v] = curl_rn(cd2, hz1.v[v], H.c[1].v[v], cd1, y2.v[v], H.c[2].v[v]);
        K.c[1].v[v] = curl_rn(cd0, xb, H.c[2].v[v], cd2, hz0.v[v], H.c[0].v[v]);
        K.c[2].v[v] = curl_rn(cd1, y0.v[v], H.c[0].v[v], cd0, xa, H.c[1].v[v]);
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        if constexpr (PV) {
          m.c[c] = lds(S + 3 * (G::E_ELEMS + G::H_ELEMS) + c * G::M_ELEMS + ha - kTmaX);
        } else {
#pragma unroll
          for (int v = 0; v < VN; ++v) m.c[c].v[v] = p.eps_scalar;
        }
      }
      if (!tf) {
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
          for (int v = 0; v < VN; ++v) E.c[c].v[v] = fma_rn(m.c[c].v[v], K.c[c].v[v], E.c[c].v[v]);
      } else {
#pragma unroll
        for (int v = 0; v < VN; ++v) {
          const bool sp = x0 + v < p.nx && ((v ? cls.y : cls.x) & kSpecialE) != 0;
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            if (sp) {  // keeps its D state
              const T t = add_rn(D.c[c].v[v], K.c[c].v[v]);
              p.D[c][q + v] = t;
              E.c[c].v[v] = mul_rn(m.c[c].v[v], t);
            } else {
              E.c[c].v[v] = fma_rn(m.c[c].v[v], K.c[c].v[v], E.c[c].v[v]);
            }
          }
        }
      }
      put3(p.En, E, 2240);
    }
    hz0 = H.c[0];
    hz1 = H.c[1];
    q += p.plane;
    if (l > 0) {
      tbits >>= 1;
      if (((k0 + l) & 63) == 0 && l < N) tbits = tile_word(k0 + l);
    }
    // every thread is done with load l: its stage takes load l + kFusedStages
    fence_proxy_async();
    __syncthreads();
    if (issuer && gave_up < 0 && l + kFusedStages < N + 2) issue(l + kFusedStages, st);
    st = sn;
    parity = pn;
  }
  // an issuer that gave up waits (bounded) for the copies it has in flight
  if (issuer && gave_up >= 0)
    for (int l = gave_up; l < min(gave_up + kFusedStages, N + 2); ++l)
      mbar_wait_sleep(smem_u32(bars + (l - l0) % kFusedStages), uint32_t(((l - l0) / kFusedStages) & 1),
                      kLimit);
}

// The ring around the grid (ghost and wall layers) from one set into the other, one
// thread per element: the two x faces with their edges, the y faces with theirs along
// z, the z faces.
template <typename T>
__global__ void __launch_bounds__(256) mirror_ring_kernel(const RingArgs<T> a) {
  const T* from = a.from[blockIdx.y];
  T* to = a.to[blockIdx.y];
  const long long fx = 2ll * (a.ny + 2) * (a.nz + 2), fy = 2ll * a.nx * (a.nz + 2), fz = 2ll * a.nx * a.ny;
  for (long long u = blockIdx.x * 256ll + threadIdx.x; u < fx + fy + fz; u += gridDim.x * 256ll) {
    int x, y, z;
    if (u < fx) {
      const long long e = u >> 1;
      x = u & 1 ? a.nx : -1;
      y = int(e % (a.ny + 2)) - 1;
      z = int(e / (a.ny + 2)) - 1;
    } else if (u < fx + fy) {
      const long long e = u - fx, r = e / a.nx;
      x = int(e % a.nx);
      y = r & 1 ? a.ny : -1;
      z = int(r >> 1) - 1;
    } else {
      const long long e = u - fx - fy, r = e / a.nx;
      x = int(e % a.nx);
      y = int(r % a.ny);
      z = r >= a.ny ? a.nz : -1;
    }
    const long long q = a.origin + z * a.plane + y * a.pitch + x;
    if (KH_IN(q, a.total, 2250)) to[q] = from[q];
  }
}

template <typename T>
void launch_mirror_ring(const RingArgs<T>& a, void* stream) {
  const long long n = 2ll * (a.ny + 2) * (a.nz + 2) + 2ll * a.nx * (a.nz + 2) + 2ll * a.nx * a.ny;
  const dim3 grid(unsigned(std::min<long long>((n + 255) / 256, 1 << 20)), 6);
  mirror_ring_kernel<T><<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(a);
}

template <typename T>
void launch_step_fused(const FusedParams<T>& p, const FusedMaps& maps, void* stream) {
  const dim3 block(32, kFusedRows, 1);
  const dim3 grid((p.nx + p.tile_w - 1) / p.tile_w, (p.ny + kFusedRows - 2) / (kFusedRows - 1),
                  (p.nz + p.zplanes - 1) / p.zplanes);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (p.stall_tx) {
    if (p.pervox_eps) step_fused_kernel<T, true, true><<<grid, block, FusedGeom<T, true>::SMEM, st>>>(p, maps);
    else step_fused_kernel<T, false, true><<<grid, block, FusedGeom<T, false>::SMEM, st>>>(p, maps);
    return;
  }
  if (p.pervox_eps) step_fused_kernel<T, true><<<grid, block, FusedGeom<T, true>::SMEM, st>>>(p, maps);
  else step_fused_kernel<T, false><<<grid, block, FusedGeom<T, false>::SMEM, st>>>(p, maps);
}

template <typename T, bool PV, bool STALL = false>
static int set_fused_attr() {
  return int(cudaFuncSetAttribute(step_fused_kernel<T, PV, STALL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  int(FusedGeom<T, PV>::SMEM)));
}

template <typename T>
int prepare_fused_kernels() {
  return set_fused_attr<T, true>() | set_fused_attr<T, false>() | set_fused_attr<T, true, true>() |
         set_fused_attr<T, false, true>();
}

template <typename T>
int fused_resident_ctas() {
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, step_fused_kernel<T, true>, 32 * kFusedRows,
                                                    FusedGeom<T, true>::SMEM) != cudaSuccess)
    return 1;
  return n > 0 ? n : 1;
}

template void launch_step_fused<float>(const FusedParams<float>&, const FusedMaps&, void*);
template void launch_mirror_ring<float>(const RingArgs<float>&, void*);
template int prepare_fused_kernels<float>();
template int fused_resident_ctas<float>();

}  // namespace kh
