// Reduced-state half-step kernel for sm_103a: plain cells, CPML cells with
// the CUDA-path stages on the auxiliaries that do not follow from others
// (kh_lean.cuh), and special cells left to the sparse passes.
//
// A CTA owns a tile of 64 × kLeanY cells and marches its z chunk, H downwards
// and E upwards, so that the z neighbour of the curl is the plane the thread
// has just computed and stays in registers: a plane needs one ring stage.  One
// elected thread keeps kLeanStages planes of TMA tiles in flight (curl sources
// with their x/y halo, updated components, m⁻¹).
//
// What bounds it: plain tiles run at the memory's rate (216×200×168 FP32 without
// CPML, which whole steps take by default: 48 µs a half-step for 262 MB, 5.5 TB/s); tiles in the CPML by the latency
// of a plane (their auxiliaries' loads, then update, store and barrier) and its
// instructions.  Against the complete cascade (T, U, W stored for every CPML cell)
// a 320×192×128 step moves 757 instead of 978 MB, in 42 + 50 M instead of 64 + 66 M
// warp instructions.
//
// Every mbarrier wait is bounded: after kSleepWaitLimit tries the thread records
// KH_ERR_TIMEOUT, leaves its cells alone from then on, and the issuing thread
// waits (bounded) for the copies it issued before the CTA ends.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "../../include/khronos_gb300.h"
#include "kh_async.cuh"
#include "kh_lean.cuh"

namespace kh {

#ifdef KH_DEBUG_BOUNDS
KH_DBG_READER(dbg_read_lean)
#endif

namespace {

template <typename T, bool PV>
struct LeanGeom {
  static constexpr int HX = 16 / int(sizeof(T));  // x halo of the curl-source box (16 bytes)
  static constexpr int XO = xoff<T>();
  static constexpr int AX = kLeanX + HX;
  static constexpr int A_BYTES = AX * (kLeanY + 1) * int(sizeof(T));
  static constexpr int A_ELEMS = ((A_BYTES + 127) / 128 * 128) / int(sizeof(T));
  static constexpr int O_ELEMS = kLeanX * kLeanY;
  static constexpr int STAGE = 3 * A_ELEMS + (PV ? 6 : 3) * O_ELEMS;  // A0..2, O0..2(, m0..2)
  static constexpr size_t SMEM =
      size_t(kLeanStages) * STAGE * sizeof(T) + (kLeanX + kLeanZ) * sizeof(AxisCoef<T>) + kLeanStages * sizeof(uint64_t);
};

}  // namespace

constexpr int kLeanThreads = kLeanY * kLeanX / kLeanVN;

// VIEW: the first or last step of a call while the program holds views of this half's
// fields (HalfStepParams::view).  In the absorber outside the own-axis CPML O is the
// state, but a value written through a view does not belong to it; the array of T, free
// there, holds a copy of O between calls.  Such a step moves as much as the complete
// cascade does.  In FP32 with per-voxel m⁻¹ it spills at six CTAs per SM (VIEW 1), which
// small grids, all of them resident at once, bear better than fewer CTAs; others take
// five (VIEW 2).  µs a step of calls of one step, 64³ / 96³ / 160×160×96, where the copies
// no longer fit the L2: without views 26.3 / 42.5 / 75, VIEW 1 31.6 / 49.2 / 102, VIEW 2
// 31.0 / 54.3 / 93.5, the complete cascade 30.7 / 56.2 / 94.8, the copies in launches of
// their own 39.7 / 59.9 / 117.
template <typename T, bool H, bool PV, bool STALL = false, bool PER = false, int VIEW = 0>
__global__ void __launch_bounds__(kLeanThreads, (VIEW == 2 ? kLeanMinBlocks<T> - 1 : kLeanMinBlocks<T>))
    half_step_lean_kernel(const __grid_constant__ HalfStepParams<T> p, const __grid_constant__ TmaMaps maps) {
  using G = LeanGeom<T, PV>;
  constexpr int VN = kLeanVN;
  static_assert(VN == 2, "paired loads of the class words");
  // Rows in update_row's branch-free forms, except in FP32 with per-voxel m⁻¹, where
  // their longer live ranges spill at six CTAs per SM (320×192×128, 96 steps, when it was
  // chosen: 15.96 ms with update_cells in both halves, 15.37 with this choice, 15.73 with
  // update_row in both; FP64 240×144×96, where a branch costs both sides' arithmetic, 17.9
  // to 13.0).
  constexpr bool kRow = sizeof(T) == 8 || !PV;
  constexpr int LPR = kLeanX / VN;  // lanes per tile row
  using PK = Pack<T, VN>;
  constexpr int s = H ? 1 : -1;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  T* stages = reinterpret_cast<T*>(smem_raw);
  AxisCoef<T>* xtab = reinterpret_cast<AxisCoef<T>*>(stages + kLeanStages * G::STAGE);  // per tile column: a, b, om, op
  AxisCoef<T>* ztab = xtab + kLeanX;                                                    // per plane of the chunk
  uint64_t* bars = reinterpret_cast<uint64_t*>(ztab + kLeanZ);

  const int tid = threadIdx.x;
  const int col = (tid % LPR) * VN;
  const int wy = tid / LPR;
  const bool issuer = tid == 0;
  const int x_tile = blockIdx.x * kLeanX;
  const int y_tile = blockIdx.y * kLeanY;
  const int j = y_tile + wy;
  const int x0 = x_tile + col;
  const bool lane_ok = j < p.ny && x0 < p.nx;
  const bool full = x0 + VN <= p.nx;  // all VN cells exist
  const int k0 = blockIdx.z * p.zplanes;
  const int k1 = min(k0 + p.zplanes, p.nz);
  const int N = k1 - k0;
  constexpr int kLimit = STALL ? kStallSleepWaitLimit : kSleepWaitLimit;
  const bool tfx = x_tile < p.red_lo[0] || (p.red_hi[0] > 0 && x_tile + kLeanX > p.nx - p.red_hi[0]);
  const bool tfy = y_tile < p.red_lo[1] || (p.red_hi[1] > 0 && y_tile + kLeanY > p.ny - p.red_hi[1]);

  if (issuer) {
    for (int st = 0; st < kLeanStages; ++st) mbar_init(&bars[st], 1);
    mbar_fence_init();
  }
  if (tfx)
    for (int c = tid; c < kLeanX; c += kLeanThreads) {
      const int i = x_tile + c;
      const bool f = i < p.nx && (i < p.red_lo[0] || i >= p.nx - p.red_hi[0]);
      const RedAxis<T> r = red_axis<T>(f && KH_IN(i, p.nx, 2120) ? p.ax[0][i] : AxisCoef<T>{}, f);
      xtab[c] = {r.a, r.b, r.om, r.op};
    }
  if (k0 < p.red_lo[2] || k1 > p.nz - p.red_hi[2])
    for (int c = tid; c < N; c += kLeanThreads) {
      const bool f = k0 + c < p.red_lo[2] || k0 + c >= p.nz - p.red_hi[2];
      const RedAxis<T> r = red_axis<T>(f && KH_IN(k0 + c, p.nz, 2112) ? p.ax[2][k0 + c] : AxisCoef<T>{}, f);
      ztab[c] = {r.a, r.b, r.om, r.op};
    }
  __syncthreads();

  // load n: the tiles of the n-th plane of the march
  auto issue = [&](int n, int st) {
    T* dst = stages + st * G::STAGE;
    const int k = H ? k1 - 1 - n : k0 + n;
    if (STALL && n == 0) {
      // failure-detection test instantiation: the first stage expects 16 bytes
      // and no copy is issued into it, so the wait on it runs out and nothing
      // is left in flight when the CTA returns
      mbar_arrive_expect_tx(&bars[st], 16u);
      return;
    }
    mbar_arrive_expect_tx(&bars[st], 3u * uint32_t(G::A_BYTES) + (PV ? 6u : 3u) * uint32_t(G::O_ELEMS * sizeof(T)));
    const int zc = k + 1;                                        // padded plane index
    const int ax = H ? G::XO + x_tile : G::XO - G::HX + x_tile;  // padded x of the A box
    const int ay = H ? 1 + y_tile : y_tile;                      // padded y of the A box
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      tma_load_3d(dst + c * G::A_ELEMS, &maps.a[c], ax, ay, zc, &bars[st]);
      tma_load_3d(dst + 3 * G::A_ELEMS + c * G::O_ELEMS, &maps.o[c], G::XO + x_tile, 1 + y_tile, zc, &bars[st]);
      if constexpr (PV)
        tma_load_3d(dst + 3 * G::A_ELEMS + (3 + c) * G::O_ELEMS, &maps.m[c], G::XO + x_tile, 1 + y_tile, zc,
                    &bars[st]);
    }
    // the plane's y/z auxiliaries into L2 ahead of the register loads (the
    // x ones, a few columns of the tile, are fetched by their own lanes)
    const bool tfz = k < p.red_lo[2] || k >= p.nz - p.red_hi[2];
    if (tfy) tma_prefetch_3d(&maps.t[1], G::XO + x_tile, 1 + y_tile, zc);
    if (tfz) tma_prefetch_3d(&maps.t[2], G::XO + x_tile, 1 + y_tile, zc);
    if (tfy && tfz) tma_prefetch_3d(&maps.u[0], G::XO + x_tile, 1 + y_tile, zc);
  };
  if (issuer) {
    const int first = min(kLeanStages, N);
    for (int n = 0; n < first; ++n) issue(n, n);
  }

  const long long step = H ? -p.plane : p.plane;
  long long q = p.origin + (long long)(H ? k1 - 1 : k0) * p.plane + (long long)j * p.pitch + x0;
  T *o0 = p.O[0] + q, *o1 = p.O[1] + q, *o2 = p.O[2] + q;
  auto get = [&](const T* arr, int site) -> PK {
    return KH_IN(q, p.total, site) && KH_IN(q + VN - 1, p.total, site) ? *reinterpret_cast<const PK*>(arr + q) : PK{};
  };
  auto put = [&](T* a, const PK& x, int site) {
    if (full) {
      if (KH_IN(q, p.total, site) && KH_IN(q + VN - 1, p.total, site)) *reinterpret_cast<PK*>(a) = x;
    } else {
#pragma unroll
      for (int v = 0; v < VN - 1; ++v)
        if (x0 + v < p.nx && KH_IN(q + v, p.total, site)) a[v] = x.v[v];
    }
  };
  // the z neighbour plane of the first plane of the march
  PK nb0{}, nb1{};
  if (lane_ok) {
    const long long qn = q - step;
    if (KH_IN(qn, p.total, 2101) && KH_IN(qn + VN - 1, p.total, 2102)) {
      nb0 = *reinterpret_cast<const PK*>(p.A[0] + qn);
      nb1 = *reinterpret_cast<const PK*>(p.A[1] + qn);
    }
  }
  const bool fy = lane_ok && (j < p.red_lo[1] || j >= p.ny - p.red_hi[1]);
  const RedAxis<T> ry = red_axis<T>(fy && KH_IN(j, p.ny, 2111) ? p.ax[1][j] : AxisCoef<T>{}, fy);
  bool fxv[VN], anyfx = false;
#pragma unroll
  for (int v = 0; v < VN; ++v) {
    const int i = x0 + v;
    fxv[v] = tfx && lane_ok && i < p.nx && (i < p.red_lo[0] || i >= p.nx - p.red_hi[0]);
    anyfx |= fxv[v];
  }
  // VIEW: the absorber's layers with those of σ = 0
  auto in_layer = [&](int a, int i) { return i < p.pml_lo[a] || i >= p.n_axis(a) - p.pml_hi[a]; };
  bool lxv[VN] = {}, ly = false, anylx = false;
  if constexpr (VIEW != 0) {
#pragma unroll
    for (int v = 0; v < VN; ++v) {
      lxv[v] = lane_ok && x0 + v < p.nx && in_layer(0, x0 + v);
      anylx |= lxv[v];
    }
    ly = lane_ok && in_layer(1, j);
  }
  // special-cell plane bits of this row segment, one word per 64 planes
  const long long tb_group = (long long)p.ny * p.nxb;
  const long long tb_row = (long long)j * p.nxb + (x0 >> 6);
  auto tile_word = [&](int g) -> uint64_t {
    return (p.tile_bits && lane_ok && KH_IN(tb_row + g * tb_group, p.n_tile_words, 2103))
               ? p.tile_bits[tb_row + g * tb_group] : 0ull;
  };
  // the bit of the current plane is the top (H) or the bottom (E) one
  int k = H ? k1 - 1 : k0;
  auto tile_bits_from = [&](int kk) -> uint64_t {
    const uint64_t w = tile_word(kk >> 6);
    return H ? w << (63 - (kk & 63)) : w >> (kk & 63);
  };
  uint64_t tbits = tile_bits_from(k);
  const int a = (H ? wy : wy + 1) * G::AX + (H ? 0 : G::HX) + col;
  const int ob = wy * kLeanX + col;
  const T cd0 = p.cd[0], cd1 = p.cd[1], cd2 = p.cd[2];
  int gave_up = -1;  // the plane at which this thread's wait ran out
  int st = 0;        // ring stage of load n, and the parity of its phase
  uint32_t parity = 0;
  for (int n = 0; n < N; ++n) {
    const bool fz = k < p.red_lo[2] || k >= p.nz - p.red_hi[2];
    const bool tf = H ? (tbits >> 63) != 0 : (tbits & 1ull) != 0;
    const bool plain = !(anyfx || fy || fz || tf);
    const bool lz = VIEW != 0 && in_layer(2, k), layer = VIEW != 0 && (anylx || ly || lz);
    const bool all_t = tf || layer;
    // auxiliaries: T in the own-axis CPML, U in those of both other axes; rows
    // with special cells take all of them, VIEW steps all of T
    Cells<T, VN> t, u;
    if constexpr (kRow || VIEW != 0) t = u = Cells<T, VN>{};
    uint2 cls{0u, 0u};  // class words of the two cells
    auto read_cls = [&] {
      if (KH_IN(q, p.total, 2110) && KH_IN(q + VN - 1, p.total, 2110))
        cls = *reinterpret_cast<const uint2*>(p.cell_class + q);
    };
    if ((!plain || layer) && lane_ok) {
      // FP64 reads them with the auxiliaries; in FP32 their registers cost the rows
      // without special cells more (320×192×128, 96 steps: 14.97 to 15.12 ms)
      if (sizeof(T) == 8 && tf) read_cls();
      if (anyfx || all_t) t.c[0] = get(p.Ts[0], 2104);
      if (fy || all_t) t.c[1] = get(p.Ts[1], 2105);
      if (fz || all_t) t.c[2] = get(p.Ts[2], 2106);
      if (fy && (fz || tf)) u.c[0] = get(p.U[0], 2107);
      if (fz && (anyfx || tf)) u.c[1] = get(p.U[1], 2108);
      if (anyfx && (fy || tf)) u.c[2] = get(p.U[2], 2109);
      if (anyfx && n + kLeanXpf < N) {
        const long long qp = q + kLeanXpf * step;
        if (KH_IN(qp + VN - 1, p.total, 2113)) {
          l2_prefetch(p.Ts[0] + qp);
          if (fz) l2_prefetch(p.U[1] + qp);
          if (fy) l2_prefetch(p.U[2] + qp);
        }
      }
    }
    if (gave_up < 0 && !mbar_wait_sleep(smem_u32(bars + st), parity, kLimit)) {
      gave_up = n;
      if (p.err) atomicExch(p.err, KH_ERR_TIMEOUT);
    }
    const bool smem_ok = KH_IN(a + (H ? 0 : -1), G::A_ELEMS, 2114) && KH_IN(a + (H ? VN : VN - 1), G::A_ELEMS, 2115) &&
                         KH_IN(a + s * G::AX, G::A_ELEMS, 2116) && KH_IN(a + s * G::AX + VN - 1, G::A_ELEMS, 2117) &&
                         KH_IN(ob + VN - 1, G::O_ELEMS, 2118);
    if (gave_up < 0 && lane_ok && smem_ok) {
      const T* A0 = stages + st * G::STAGE + a;
      const T* A1 = A0 + G::A_ELEMS;
      const T* A2 = A1 + G::A_ELEMS;
      const T* Os = stages + st * G::STAGE + 3 * G::A_ELEMS + ob;
      auto lds = [](const T* q) { return *reinterpret_cast<const PK*>(q); };
      const PK c0 = lds(A0), c1 = lds(A1), c2 = lds(A2), y0 = lds(A0 + s * G::AX), y2 = lds(A2 + s * G::AX);
      const T e1 = A1[H ? VN : -1], e2 = A2[H ? VN : -1];  // x neighbours past the thread's cells
      Cells<T, VN> O, m, K;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        O.c[c] = lds(Os + c * G::O_ELEMS);
        if constexpr (PV) {
          m.c[c] = lds(Os + (3 + c) * G::O_ELEMS);
        } else {
#pragma unroll
          for (int v = 0; v < VN; ++v) m.c[c].v[v] = p.m_scalar;
        }
      }
#pragma unroll
      for (int v = 0; v < VN; ++v) {
        // forward difference (H): cell v reads x + 1; backward (E): x - 1
        const T x1 = H ? (v + 1 < VN ? c1.v[(v + 1) % VN] : e1) : (v > 0 ? c1.v[(v + VN - 1) % VN] : e1);
        const T x2 = H ? (v + 1 < VN ? c2.v[(v + 1) % VN] : e2) : (v > 0 ? c2.v[(v + VN - 1) % VN] : e2);
        K.c[0].v[v] = curl_rn(cd2, nb1.v[v], c1.v[v], cd1, y2.v[v], c2.v[v]);
        K.c[1].v[v] = curl_rn(cd0, x2, c2.v[v], cd2, nb0.v[v], c0.v[v]);
        K.c[2].v[v] = curl_rn(cd1, y0.v[v], c0.v[v], cd0, x1, c1.v[v]);
      }
      nb0 = c0;
      nb1 = c1;
      const AxisCoef<T> zt = ztab[k - k0];  // read where fz
      bool sp[VN] = {}, anysp = false;
      if (tf) {
        constexpr uint32_t kSp = H ? kSpecialH : kSpecialE;
        if (sizeof(T) == 4) read_cls();
#pragma unroll
        for (int v = 0; v < VN; ++v) {
          sp[v] = x0 + v < p.nx && ((v ? cls.y : cls.x) & kSp) != 0;
          anysp |= sp[v];
        }
      }
      // O is the state: a cell of a layer, outside the own-axis CPML
      auto derived = [&](int c, int v) {
        return (lxv[v] || ly || lz) && !(c == 0 ? fxv[v] : (c == 1 ? fy : fz)) && !sp[v];
      };
      if constexpr (VIEW != 0) {
        if (p.view & kViewRestore) {
#pragma unroll
          for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int v = 0; v < VN; ++v)
              if (derived(c, v)) O.c[c].v[v] = t.c[c].v[v];
        }
      }
      if (anysp) {
        Cells<T, VN> w;
        if (anyfx) w.c[0] = get(p.W[0], 2128);
        if (fy) w.c[1] = get(p.W[1], 2129);
        if (fz) w.c[2] = get(p.W[2], 2119);
        RedAxis<T> rz{false, T(1), T(1), T(1), T(1)};
        if (fz) rz = {true, zt.s, zt.om, zt.ir, zt.op};
        update_special_cells<T, VN>(sp, fxv, p.ax[0] + x0, p.ax[1] + j, fz ? p.ax[2][k].s : T(0), xtab + col, ry, rz, K,
                                    m, O, t, u, w);
        if (anyfx) put(p.W[0] + q, w.c[0], 2131);
        if (fy) put(p.W[1] + q, w.c[1], 2132);
        if (fz) put(p.W[2] + q, w.c[2], 2133);
      } else {
        const AxisCoef<T>* xt = xtab + col;
        if constexpr (kRow) {
          switch ((tfx ? 1 : 0) | (fy ? 2 : 0) | (fz ? 4 : 0)) {
            case 0: update_row<false, false, false, T, VN>(fxv, xt, ry, zt, K, m, O, t, u); break;
            case 1: update_row<true, false, false, T, VN>(fxv, xt, ry, zt, K, m, O, t, u); break;
            case 2: update_row<false, true, false, T, VN>(fxv, xt, ry, zt, K, m, O, t, u); break;
            case 3: update_row<true, true, false, T, VN>(fxv, xt, ry, zt, K, m, O, t, u); break;
            case 4: update_row<false, false, true, T, VN>(fxv, xt, ry, zt, K, m, O, t, u); break;
            case 5: update_row<true, false, true, T, VN>(fxv, xt, ry, zt, K, m, O, t, u); break;
            case 6: update_row<false, true, true, T, VN>(fxv, xt, ry, zt, K, m, O, t, u); break;
            case 7: update_row<true, true, true, T, VN>(fxv, xt, ry, zt, K, m, O, t, u); break;
          }
        } else {
          RedAxis<T> rz{false, T(1), T(1), T(1), T(1)};
          if (fz) rz = {true, zt.s, zt.om, zt.ir, zt.op};
          if (plain) {
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
              for (int v = 0; v < VN; ++v) O.c[c].v[v] = fma_rn(m.c[c].v[v], K.c[c].v[v], O.c[c].v[v]);
          } else {
            update_cells<T, VN>(fxv, anyfx, xt, ry, rz, K, m, O, t, u);
          }
        }
      }
      if constexpr (VIEW != 0) {
        if (p.view & kViewKeep) {
#pragma unroll
          for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int v = 0; v < VN; ++v)
              if (derived(c, v)) t.c[c].v[v] = O.c[c].v[v];
        }
      }
      if (!plain || layer) {
        // what was loaded goes back (values that a cell does not use unchanged)
        if (anyfx || all_t) put(p.Ts[0] + q, t.c[0], 2121);
        if (fy || all_t) put(p.Ts[1] + q, t.c[1], 2122);
        if (fz || all_t) put(p.Ts[2] + q, t.c[2], 2123);
        if (fy && (fz || tf)) put(p.U[0] + q, u.c[0], 2124);
        if (fz && (anyfx || tf)) put(p.U[1] + q, u.c[1], 2125);
        if (anyfx && (fy || tf)) put(p.U[2] + q, u.c[2], 2126);
      }
      if (full) {
        if (KH_IN(q, p.total, 2127) && KH_IN(q + VN - 1, p.total, 2127)) {
          *reinterpret_cast<PK*>(o0) = O.c[0];
          *reinterpret_cast<PK*>(o1) = O.c[1];
          *reinterpret_cast<PK*>(o2) = O.c[2];
        }
      } else {
        put(o0, O.c[0], 2127);
        put(o1, O.c[1], 2127);
        put(o2, O.c[2], 2127);
      }
      if constexpr (PER) {
        // periodic axes: the face cells also into the ghost layer across (layer 0
        // into n, layer n - 1 into -1, over the cells of the other two axes), instead
        // of a wrap launch after each half (256×256×128, x and y, 64 steps: 10.96 to
        // 10.04 ms; 64³ 21.5 to 17.5 µs a step)
        if ((p.wrap & 1u) && (x0 == 0 || x0 + VN >= p.nx)) {
          T* const o[3] = {o0, o1, o2};
#pragma unroll
          for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int v = 0; v < VN; ++v) {
              if (x0 + v == 0 && KH_IN(q + p.nx, p.total, 2140)) o[c][p.nx] = O.c[c].v[v];
              if (x0 + v == p.nx - 1 && KH_IN(q + v - p.nx, p.total, 2141)) o[c][v - p.nx] = O.c[c].v[v];
            }
        }
        auto across = [&](bool lo, bool hi, long long d) {
          if (lo && KH_IN(q + d + VN - 1, p.total, 2142)) {
            put(o0 + d, O.c[0], 2143);
            put(o1 + d, O.c[1], 2143);
            put(o2 + d, O.c[2], 2143);
          }
          if (hi && KH_IN(q - d, p.total, 2144)) {
            put(o0 - d, O.c[0], 2145);
            put(o1 - d, O.c[1], 2145);
            put(o2 - d, O.c[2], 2145);
          }
        };
        if (p.wrap & 2u) across(j == 0, j == p.ny - 1, (long long)p.ny * p.pitch);
        if (p.wrap & 4u) across(k == 0, k == p.nz - 1, (long long)p.nz * p.plane);
      }
    }
    q += step;
    o0 += step;
    o1 += step;
    o2 += step;
    // every thread is done with load n: its stage takes load n + kLeanStages
    __syncthreads();
    if (issuer && gave_up < 0 && n + kLeanStages < N) {
      fence_proxy_async();
      issue(n + kLeanStages, st);
    }
    if (++st == kLeanStages) {
      st = 0;
      parity ^= 1u;
    }
    k += H ? -1 : 1;
    tbits = H ? tbits << 1 : tbits >> 1;
    if ((k & 63) == (H ? 63 : 0) && n + 1 < N) tbits = tile_bits_from(k);
  }
  // an issuer that gave up waits (bounded) for the copies it has in flight
  if (issuer && gave_up >= 0)
    for (int l = gave_up; l < min(gave_up + kLeanStages, N); ++l)
      mbar_wait_sleep(smem_u32(bars + l % kLeanStages), uint32_t((l / kLeanStages) & 1), kLimit);
}

// ---------------------------------------------------------------------------
// The CPML axes of a cell (layers of σ = 0 at its inner edge count as outside); whether
// it lies in a layer at all, where the complete state has T.
template <typename T>
__device__ __forceinline__ bool in_absorber(const HalfStepParams<T>& p, int i, int j, int k, bool (&f)[3]) {
  const int at[3] = {i, j, k};
  bool any = false;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    f[a] = at[a] < p.red_lo[a] || at[a] >= p.n_axis(a) - p.red_hi[a];
    any |= at[a] < p.pml_lo[a] || at[a] >= p.n_axis(a) - p.pml_hi[a];
  }
  return any;
}

// The complete T, U, W of every CPML cell from the reduced state, for state
// files and for the general kernel (kh_lean.cuh says how they follow).
template <typename T, bool H>
__global__ void expand_state_kernel(const HalfStepParams<T> p, bool o_kept) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= p.nx) return;
  for (int k = blockIdx.z; k < p.nz; k += gridDim.z)
    for (int j = blockIdx.y; j < p.ny; j += gridDim.y) {
      bool f[3];
      if (!in_absorber(p, i, j, k, f)) continue;
      const long long q = p.origin + (long long)k * p.plane + (long long)j * p.pitch + i;
      if (!KH_IN(q, p.total, 2130)) continue;
      if (p.cell_class && (p.cell_class[q] & (H ? kSpecialH : kSpecialE))) continue;  // keeps the complete state
      const int idx[3] = {i, j, k};
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const int n = (c + 1) % 3, v = (c + 2) % 3;
        const T m = p.m_inv[c] ? p.m_inv[c][q] : p.m_scalar;
        const T t = f[c] ? p.Ts[c][q] : derived_t(o_kept ? p.Ts[c][q] : p.O[c][q], m);
        p.Ts[c][q] = t;
        if (f[n] && !f[v] && p.ax[n][idx[n]].s != T(0)) p.U[c][q] = t;
        if (f[c] && p.ax[c][idx[c]].s != T(0)) p.W[c][q] = mul_rn(m, t);
      }
    }
}

// One thread per cell; further rows and planes in turn above the grid's limits.
template <typename T>
static dim3 cell_grid(const HalfStepParams<T>& p) {
  return dim3((p.nx + 127) / 128, std::min(p.ny, 65535), std::min(p.nz, 65535));
}

template <typename T>
void launch_expand_state(bool h_half, const HalfStepParams<T>& p, bool o_kept, void* stream) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (h_half) expand_state_kernel<T, true><<<cell_grid(p), 128, 0, st>>>(p, o_kept);
  else expand_state_kernel<T, false><<<cell_grid(p), 128, 0, st>>>(p, o_kept);
}

// Cell u of the layers: its indices and its place in the padded arrays.
template <typename T>
__device__ __forceinline__ long long layer_cell(const KeepArgs<T>& a, long long u, int (&at)[3]) {
  int b = 0;
  while (u >= a.first[b + 1]) ++b;
  const long long e = u - a.first[b];
  if (e <= 0xffffffffll) {  // 32-bit division wherever the index fits
    const unsigned r = unsigned(e) / unsigned(a.dims[b][0]);
    at[0] = a.start[b][0] + int(unsigned(e) - r * unsigned(a.dims[b][0]));
    at[2] = a.start[b][2] + int(r / unsigned(a.dims[b][1]));
    at[1] = a.start[b][1] + int(r % unsigned(a.dims[b][1]));
  } else {
    const long long r = e / a.dims[b][0];
    at[0] = a.start[b][0] + int(e % a.dims[b][0]);
    at[2] = a.start[b][2] + int(r / a.dims[b][1]);
    at[1] = a.start[b][1] + int(r % a.dims[b][1]);
  }
  return a.origin + at[2] * a.plane + at[1] * a.pitch + at[0];
}

// O of the CPML cells where it is the state into the array of T, free there (KeepArgs):
// one thread per cell of the absorber's layers.
template <typename T>
__global__ void __launch_bounds__(256) keep_state_kernel(const __grid_constant__ KeepArgs<T> a, bool from_t) {
  const KeepHalf<T>& h = a.half[blockIdx.y];
  for (long long u = blockIdx.x * 256ll + threadIdx.x; u < a.first[6]; u += gridDim.x * 256ll) {
    int at[3];
    const long long q = layer_cell(a, u, at);
    if (!KH_IN(q, a.total, 2151)) continue;
    if (h.tile_bits) {  // special cells keep their T
      const long long w = ((long long)(at[2] >> 6) * a.n[1] + at[1]) * a.nxb + (at[0] >> 6);
      if (((h.tile_bits[w] >> (at[2] & 63)) & 1ull) && (a.cell_class[q] & h.special)) continue;
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      if (at[c] < h.lo[c] || at[c] >= a.n[c] - h.hi[c]) continue;  // T is the state
      const T o = h.O[c][q];
      if (!from_t) {
        h.Ts[c][q] = o;
      } else {
        const T mt = mul_rn(h.m_inv[c] ? h.m_inv[c][q] : h.m_scalar, h.Ts[c][q]);
        h.Ts[c][q] = fabs(o - mt) <= derived_tol(mt) ? o : mt;
      }
    }
  }
}

template <typename T>
void launch_keep_state(const KeepArgs<T>& a, int halves, bool from_t, void* stream) {
  if (a.first[6] <= 0) return;
  const dim3 grid(unsigned(std::min<long long>((a.first[6] + 255) / 256, 1 << 30)), unsigned(halves));
  keep_state_kernel<T><<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(a, from_t);
}

// Cells of the layers where O is the state and m⁻¹ = 0: T does not follow from a field
// that is zero, so they keep it as special cells do.  Without cls: are there any?
template <typename T>
__global__ void __launch_bounds__(256) dead_cells_kernel(const __grid_constant__ KeepArgs<T> a, uint32_t* cls, int* found) {
  const KeepHalf<T>& h = a.half[blockIdx.y];
  for (long long u = blockIdx.x * 256ll + threadIdx.x; u < a.first[6]; u += gridDim.x * 256ll) {
    int at[3];
    const long long q = layer_cell(a, u, at);
    if (!KH_IN(q, a.total, 2152)) continue;
    bool dead = false;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const bool derived = !(at[c] < h.lo[c] || at[c] >= a.n[c] - h.hi[c]);
      dead |= derived && h.m_inv[c] && h.m_inv[c][q] == T(0);
    }
    if (!dead) continue;
    if (cls) atomicOr(cls + q, h.special);
    else *found = 1;
  }
}

template <typename T>
void launch_dead_cells(const KeepArgs<T>& a, int halves, uint32_t* cls, int* found, void* stream) {
  if (a.first[6] <= 0) return;
  const dim3 grid(unsigned(std::min<long long>((a.first[6] + 255) / 256, 1 << 30)), unsigned(halves));
  dead_cells_kernel<T><<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(a, cls, found);
}

// What the reduced state takes for granted, checked on the complete T, U and W of a
// state from elsewhere (StateCheck, kh_kernels.cuh).
template <typename T, bool H>
__global__ void check_state_kernel(const HalfStepParams<T> p, StateCheck<T>* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= p.nx) return;
  bool broken = false;
  T top_t = T(0), off_u = T(0), top_o = T(0), off_o = T(0);
  // the largest so far; NaN counts as infinite
  auto most = [](T& m, T x) {
    if (!(x <= m)) m = x == x ? x : T(INFINITY);
  };
  for (int k = blockIdx.z; k < p.nz; k += gridDim.z)
    for (int j = blockIdx.y; j < p.ny; j += gridDim.y) {
      bool f[3];
      if (!in_absorber(p, i, j, k, f)) continue;
      const long long q = p.origin + (long long)k * p.plane + (long long)j * p.pitch + i;
      if (!KH_IN(q, p.total, 2150)) continue;
      if (p.cell_class && (p.cell_class[q] & (H ? kSpecialH : kSpecialE))) continue;  // keeps the complete state
      const int idx[3] = {i, j, k};
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const int n = (c + 1) % 3, v = (c + 2) % 3;
        const T t = p.Ts[c][q], o = p.O[c][q];
        const T mt = mul_rn(p.m_inv[c] ? p.m_inv[c][q] : p.m_scalar, t);
        const T near = derived_tol(mt);
        if (f[c] && p.ax[c][idx[c]].s != T(0)) {
          broken |= !(fabs(p.W[c][q] - mt) <= near);
        } else if (!f[c]) {
          broken |= !(fabs(o - mt) <= near);
        } else {  // σ = 0: O goes on by differences, apart from m·T by their rounding
          most(top_o, fabs(o));
          most(off_o, fabs(o - mt));
        }
        if (f[n] && !f[v] && p.ax[n][idx[n]].s != T(0)) {
          most(top_t, fabs(t));
          most(off_u, fabs(p.U[c][q] - t));
        }
      }
    }
  if (broken) atomicOr(&out->broken, 1);
  auto raise = [](T* a, T x) {  // non-negative values order like their bits
    if constexpr (sizeof(T) == 4) atomicMax(reinterpret_cast<int*>(a), __float_as_int(x));
    else atomicMax(reinterpret_cast<long long*>(a), __double_as_longlong(x));
  };
  if (top_t > T(0)) raise(&out->top_t, top_t);
  if (off_u > T(0)) raise(&out->off_u, off_u);
  if (top_o > T(0)) raise(&out->top_o, top_o);
  if (off_o > T(0)) raise(&out->off_o, off_o);
}

template <typename T>
void launch_check_state(bool h_half, const HalfStepParams<T>& p, StateCheck<T>* out, void* stream) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (h_half) check_state_kernel<T, true><<<cell_grid(p), 128, 0, st>>>(p, out);
  else check_state_kernel<T, false><<<cell_grid(p), 128, 0, st>>>(p, out);
}

// VIEW forms: the second where the first spills.
template <typename T, bool PV>
constexpr int view_forms() {
  return sizeof(T) == 4 && PV ? 2 : 1;
}

template <typename T, bool H, bool PV, int VIEW>
static void launch_view(dim3 grid, dim3 block, const HalfStepParams<T>& p, const TmaMaps& maps, cudaStream_t st) {
  constexpr size_t smem = LeanGeom<T, PV>::SMEM;
  if (p.wrap) half_step_lean_kernel<T, H, PV, false, true, VIEW><<<grid, block, smem, st>>>(p, maps);
  else half_step_lean_kernel<T, H, PV, false, false, VIEW><<<grid, block, smem, st>>>(p, maps);
}

template <typename T, bool H, bool PV>
static void launch_lean_variant(const HalfStepParams<T>& p, const TmaMaps& maps, cudaStream_t st) {
  const dim3 block(kLeanThreads, 1, 1);
  const dim3 grid((p.nx + kLeanX - 1) / kLeanX, (p.ny + kLeanY - 1) / kLeanY, (p.nz + p.zplanes - 1) / p.zplanes);
  if constexpr (sizeof(T) == 4) {
    if (p.stall_tx) {  // failure-detection test instantiation (FP32 only)
      half_step_lean_kernel<T, H, PV, true><<<grid, block, LeanGeom<T, PV>::SMEM, st>>>(p, maps);
      return;
    }
  }
  if (p.view) {
    if constexpr (view_forms<T, PV>() == 2) {
      if (p.view_form == 2) {
        launch_view<T, H, PV, 2>(grid, block, p, maps, st);
        return;
      }
    }
    launch_view<T, H, PV, 1>(grid, block, p, maps, st);
    return;
  }
  if (p.wrap) half_step_lean_kernel<T, H, PV, false, true><<<grid, block, LeanGeom<T, PV>::SMEM, st>>>(p, maps);
  else half_step_lean_kernel<T, H, PV><<<grid, block, LeanGeom<T, PV>::SMEM, st>>>(p, maps);
}

template <typename T>
void launch_half_step_lean(bool h_half, const HalfStepParams<T>& p, const TmaMaps& maps, void* stream) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool pv = p.m_inv[0] != nullptr;
  if (h_half) {
    if (pv) launch_lean_variant<T, true, true>(p, maps, st);
    else launch_lean_variant<T, true, false>(p, maps, st);
  } else {
    if (pv) launch_lean_variant<T, false, true>(p, maps, st);
    else launch_lean_variant<T, false, false>(p, maps, st);
  }
}

template <typename T, bool H, bool PV, bool STALL = false, bool PER = false, int VIEW = 0>
static int set_lean_attr() {
  return int(cudaFuncSetAttribute(half_step_lean_kernel<T, H, PV, STALL, PER, VIEW>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  int(LeanGeom<T, PV>::SMEM)));
}

template <typename T, bool PV, int VIEW>
static int set_view_attr() {
  return set_lean_attr<T, true, PV, false, false, VIEW>() | set_lean_attr<T, true, PV, false, true, VIEW>() |
         set_lean_attr<T, false, PV, false, false, VIEW>() | set_lean_attr<T, false, PV, false, true, VIEW>();
}

template <typename T>
int prepare_lean_kernels() {
  int e = 0;
  e |= set_lean_attr<T, true, true>();
  e |= set_lean_attr<T, true, false>();
  e |= set_lean_attr<T, false, true>();
  e |= set_lean_attr<T, false, false>();
  e |= set_lean_attr<T, true, true, false, true>();
  e |= set_lean_attr<T, true, false, false, true>();
  e |= set_lean_attr<T, false, true, false, true>();
  e |= set_lean_attr<T, false, false, false, true>();
  e |= set_view_attr<T, true, 1>() | set_view_attr<T, false, 1>();
  if constexpr (sizeof(T) == 4) {
    e |= set_view_attr<T, true, 2>();
    e |= set_lean_attr<T, true, true, true>();
    e |= set_lean_attr<T, true, false, true>();
    e |= set_lean_attr<T, false, true, true>();
    e |= set_lean_attr<T, false, false, true>();
  }
  return e;
}

template <typename T>
int lean_resident_ctas(int view) {
  auto resident = [](auto kernel) {
    int n = 0;
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, kLeanThreads, LeanGeom<T, true>::SMEM);
    return e == cudaSuccess && n > 0 ? n : 1;
  };
  if (view == 2 && sizeof(T) == 4) return resident(half_step_lean_kernel<T, false, true, false, false, sizeof(T) == 4 ? 2 : 1>);
  return view ? resident(half_step_lean_kernel<T, false, true, false, false, 1>) : resident(half_step_lean_kernel<T, false, true>);
}

template void launch_half_step_lean<float>(bool, const HalfStepParams<float>&, const TmaMaps&, void*);
template void launch_half_step_lean<double>(bool, const HalfStepParams<double>&, const TmaMaps&, void*);
template void launch_expand_state<float>(bool, const HalfStepParams<float>&, bool, void*);
template void launch_expand_state<double>(bool, const HalfStepParams<double>&, bool, void*);
template void launch_keep_state<float>(const KeepArgs<float>&, int, bool, void*);
template void launch_keep_state<double>(const KeepArgs<double>&, int, bool, void*);
template void launch_dead_cells<float>(const KeepArgs<float>&, int, uint32_t*, int*, void*);
template void launch_dead_cells<double>(const KeepArgs<double>&, int, uint32_t*, int*, void*);
template void launch_check_state<float>(bool, const HalfStepParams<float>&, StateCheck<float>*, void*);
template void launch_check_state<double>(bool, const HalfStepParams<double>&, StateCheck<double>*, void*);
template int prepare_lean_kernels<float>();
template int prepare_lean_kernels<double>();
template int lean_resident_ctas<float>(int);
template int lean_resident_ctas<double>(int);

}  // namespace kh
