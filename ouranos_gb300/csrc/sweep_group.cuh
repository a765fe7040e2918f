// The sweep with H lanes to a cell: the default form of the orders above 2-D Q2 and
// 3-D Q1, and of 2-D Q2 with few cells or many materials side by side.
//
// A task is one direction crossing a tile of G = 32 / H cells of the transverse
// plane; lane (g, h) works on cell g = (lx, ly) and, at step s, on plane
// sc = s - lx - ly of the sweep axis (the skewed wavefront of sweep.cuh, whose
// canonical orientation, tickets, edge words and bounded waits are used
// unchanged).  The H lanes of a cell share all of its work, and the warp passes
// everything through its own shared-memory slot:
//   faces    lane h forms the rows t = h, h + H, ... of each inflow face's
//            product F_a psi_up,a; psi_up is read from the upwind neighbour's
//            solution of the step before (a ghost slot holds the values that
//            came through the edge words, or the boundary's);
//   b        lane h assembles the dofs i = h, h + H, ...: the source value and,
//            one after the other, its x, sweep-axis and y face terms;
//   x        lane h computes the rows i = h, h + H, ... of A'^-1 b, the two (or
//            four) values of b in 16 bytes read once for all of its rows;
//   then the outflow of the tile's last cells is published and psi stored, H
//   consecutive dofs of a cell per store.
// Every dof is rounded in the order of the per-lane and the one-warp-per-cell
// forms, whatever H is, so all forms give the same bits.
#pragma once

#include <type_traits>

#include "pack2.cuh"
#include "sweep.cuh"

namespace ouranos {

// cells of a tile: G = 32 / H along x in 2-D, WX x WY in 3-D
template <int DIM, int H>
struct GroupTile {
  static constexpr int G = 32 / H;
  static constexpr int WX = DIM == 2 ? G : (G >= 8 ? 4 : (G >= 2 ? 2 : 1));
  static constexpr int WY = G / WX;
};

// Which rows a lane owns, and the layout of the inverse tables that follows.
// Where they come out even (P1 even, N / 2 a multiple of H): pairs of dofs that are
// neighbours along x, pair m = h + H p being the rows 2m and 2m + 1 (a mirrored
// axis swaps a pair, or moves it whole).  Else the rows h + H k, taken two at a
// time, the last one alone when their number R is odd.  A matrix is stored
// [pair p][piece c][lane h] in 16-byte pieces of 16 / (2 sizeof(real)) columns of a
// row pair, then [piece c][lane h] of 16 / sizeof(real) columns of the lone row;
// what does not exist is zero.
template <int DIM, int P1, int H>
struct GroupRows {
  static constexpr int N = Cell<DIM, P1>::N;
  static constexpr bool kAdj = P1 % 2 == 0 && (N / 2) % H == 0;
  static constexpr int R = kAdj ? N / H : (N + H - 1) / H;
  static constexpr int RP = R / 2;
  static constexpr bool kOdd = R % 2 != 0;
  __host__ __device__ static constexpr int row(int h, int k) {
    return kAdj ? 2 * (h + H * (k / 2)) + k % 2 : h + H * k;
  }
  // bytes of a matrix for values of sz bytes
  __host__ __device__ static constexpr int pair_pieces(int sz) { return (N + 8 / sz - 1) / (8 / sz); }
  __host__ __device__ static constexpr int lone_pieces(int sz) { return (N + 16 / sz - 1) / (16 / sz); }
  __host__ __device__ static constexpr int matrix_bytes(int sz) {
    return 16 * H * (RP * pair_pieces(sz) + (kOdd ? lone_pieces(sz) : 0));
  }
};

// Layout of one warp's shared-memory slot (bytes)
template <typename real, int DIM, int P1, int H>
struct GroupSlot {
  using C = Cell<DIM, P1>;
  using T = GroupTile<DIM, H>;
  static constexpr int N = C::N, FD = C::FD, G = T::G;
  static constexpr int SZ = (int)sizeof(real);
  static constexpr int DB = 2 * SZ;                 // a row pair's two values
  // A cell's values start at any multiple of GR bytes: CH aligned 16-byte
  // pieces cover them wherever they start
  static constexpr int CELLB = N * SZ;
  static constexpr int GR = (CELLB & -CELLB) < 16 ? (CELLB & -CELLB) : 16;
  static constexpr int CH = (CELLB + 16 - GR + 15) / 16;
  static_assert(16 * CH - CELLB <= (int)kSrcSlack, "the sources' buffers hold the last piece");
  // strides of odd multiples of 16 bytes: the cells of a warp start on different banks
  static constexpr int SRC = 16 * (CH | 1);
  static constexpr int VEC = 16 * (((N * SZ + 15) / 16) | 1);
  static constexpr int FACE = 16 * (((DIM * FD * SZ + 15) / 16) | 1);
  static constexpr int PF = 2;                      // planes in flight ahead of the one being solved
  static constexpr int RING = PF + 1;
  static constexpr int GHOST = T::WY + (DIM == 3 ? T::WX : 0);
  static constexpr int o_f = (G + GHOST) * VEC;
  static constexpr int o_cls = o_f + G * FACE;
  static constexpr int o_src = o_cls + ((RING * G * 4 + 15) & ~15);
  // arrays streamed: q, or T and (with a fixed source) the isotropic source
  __host__ __device__ static constexpr int bytes(int arrays) { return o_src + RING * arrays * G * SRC; }
};

// 16 bytes of shared memory
template <typename real, int NV>
__device__ __forceinline__ void load_row_shared(const unsigned char* p, real (&o)[NV]) {
  constexpr int W = Bits<real>::W;
  const uint4 u = *reinterpret_cast<const uint4*>(p);
  const unsigned w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int t = 0; t < NV; ++t) o[t] = from_words<real>(w[t * W], W == 2 ? w[t * W + 1] : 0u);
}

// One tagged word: poll until its tag matches, as fetch_edge does
static __device__ __forceinline__ bool poll_word(const unsigned long long* w, unsigned tag, unsigned* out, int* status,
                                                 long long limit_ns) {
  const long long t0 = global_ns();
  unsigned sleep_ns = 16;
  for (unsigned it = 0; it < (1u << 26); ++it) {
    const unsigned long long v = ld_relaxed_u64(w);
    if ((unsigned)(v >> 32) == tag) {
      *out = (unsigned)v;
      return true;
    }
    if (it >= 8) {
      __nanosleep(sleep_ns);
      if (sleep_ns < 256) sleep_ns <<= 1;
    }
    if (*(volatile int*)status) return false;
    if (global_ns() - t0 > limit_ns) break;
  }
  atomicCAS(status, 0, 1);
  return false;
}

template <typename real, int DIM, int P1, int FM, int H>
__device__ __forceinline__ void sweep_group_task(const SweepArgs<real>& a, const int task, unsigned char* smem_raw) {
  using S = GroupSlot<real, DIM, P1, H>;
  using RW = GroupRows<DIM, P1, H>;
  using C = Cell<DIM, P1>;
  using A = Arith<real>;
  using K = Pk<real>;
  using P = typename K::P;
  using TL = GroupTile<DIM, H>;
  constexpr int N = S::N, FD = S::FD, G = S::G, SZ = S::SZ, DB = S::DB;
  constexpr int R = RW::R, RP = RW::RP;
  constexpr bool kAdj = RW::kAdj, kOdd = RW::kOdd;
  constexpr int W = Tagged<real>::W;
  constexpr int WX = TL::WX, WY = TL::WY;
  constexpr int AS = DIM - 1;               // physical axis of the sweep direction
  constexpr int KF = kAdj ? 2 * ((FD / 2 + H - 1) / H) : (FD + H - 1) / H;  // rows of a face product per lane
  constexpr int KE = (FD * W + H - 1) / H;  // edge words per lane
  constexpr int KC = (S::CH + H - 1) / H;   // 16-byte pieces of a cell's source per lane
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int h = lane % H, g = lane / H;
  const int lx = g % WX, ly = g / WX;
  const int arrays = FM == 0 ? 1 : (a.iso ? 2 : 1);
  unsigned char* sm = smem_raw + (threadIdx.x >> 5) * S::bytes(arrays);
  unsigned char* s_x = sm + g * S::VEC;                // this cell: psi of the last step, then b
  unsigned char* s_gx = sm + (G + ly) * S::VEC;        // ghost cell of the tile's x edge
  unsigned char* s_gy = sm + (G + WY + (DIM == 3 ? lx : 0)) * S::VEC;
  unsigned char* s_f = sm + S::o_f + g * S::FACE;
  const unsigned char* up_x = lx > 0 ? s_x - S::VEC : s_gx;
  const unsigned char* up_y = DIM == 3 ? (ly > 0 ? s_x - WX * S::VEC : s_gy) : nullptr;
  auto put = [](unsigned char* p, int i, real v) { *reinterpret_cast<real*>(p + i * SZ) = v; };
  auto get = [](const unsigned char* p, int i) { return *reinterpret_cast<const real*>(p + i * SZ); };
  const f2 z = f2_make(a.minus_zero, a.minus_zero);

  const int tiles = a.tiles_x * a.tiles_y;
  const int NS = a.n_sweep, NX = a.nx, NY = DIM == 3 ? a.ny : 1;
  const unsigned want_epoch = (a.epoch ^ (a.wait_bias ? 0x8000u : 0u)) << 16;
  const int2 tk = a.tasks[task];
  const int tile = tk.y;
  const int tx = tile % a.tiles_x, ty = tile / a.tiles_x;
  const int d = a.group_dirs[tk.x];  // one direction per task
  const int flip = a.group_flip[tk.x];
  const real wX = a.abs_omega[d * 3 + 0];
  const real wY = DIM == 3 ? a.abs_omega[d * 3 + 1] : real(0);
  const real wS = a.abs_omega[d * 3 + AS];
  // Inflow: a.bnd is a table of zeros where there is none, so that every call takes the
  // same path, and the values pass through a shuffle, which the whole warp waits for
  const real bX = A::shfl(a.bnd[d * 3 + 0], 0);
  const real bY = DIM == 3 ? A::shfl(a.bnd[d * 3 + 1], 0) : real(0);
  const real bS = A::shfl(a.bnd[d * 3 + AS], 0);
  real w0 = 0;
  if (FM >= 1) w0 = a.m2d[(size_t)d * a.n_mom];
  // physical position of canonical dof i: base + c0 st0 + c1 st1 + c2 st2
  int base = 0, st0 = 1, st1 = P1, st2 = P1 * P1;
  if (flip & 1) { base += P1 - 1; st0 = -1; }
  if (flip & 2) { base += (P1 - 1) * P1; st1 = -P1; }
  if (DIM == 3 && (flip & 4)) { base += (P1 - 1) * P1 * P1; st2 = -P1 * P1; }
  const bool swap = kAdj && (flip & 1);  // a pair's two dofs change places
  // physical position of this lane's dofs (even P1: of its pairs' first)
  int po[kAdj ? RP : R];
#pragma unroll
  for (int k = 0; k < (kAdj ? RP : R); ++k) {
    const int i0 = RW::row(h, kAdj ? 2 * k : k);
    const int i = i0 < N ? i0 : 0;
    po[k] = base + C::comp(i, 0) * st0 + C::comp(i, 1) * st1 + (DIM == 3 ? C::comp(i, 2) * st2 : 0) - (swap ? 1 : 0);
  }
  const int xc = tx * WX + lx, yc = ty * WY + ly;  // canonical column
  const bool col_ok = xc < NX && (DIM == 2 || yc < NY);
  const int xp = (flip & 1) ? NX - 1 - xc : xc;
  const int yp = DIM == 3 ? ((flip & 2) ? NY - 1 - yc : yc) : 0;
  const int sflip = DIM == 3 ? (flip & 4) : (flip & 2);
  const long plane = DIM == 2 ? (long)NX : (long)NX * NY;
  const long cstep = sflip ? -plane : plane;  // cells from one step to the next
  // cell of step 0 (outside the mesh before the column's first step: the
  // pointers below walk in from there and are used on its planes only)
  long cell = (long)xp + (long)NX * yp + (sflip ? plane * (NS - 1) : 0) - cstep * (lx + ly);
  const size_t dirbase = (size_t)d * a.n_dofs;
  const unsigned char* ainv = reinterpret_cast<const unsigned char*>(a.ainv) +
                              (size_t)a.dir_class[d] * RW::matrix_bytes(SZ) + 16 * h;
  const size_t ainv_class = (size_t)a.n_dir_class * RW::matrix_bytes(SZ);
  const real* src0 = FM == 0 ? a.q + dirbase : a.src;

  // the source of step `st` into ring slot `slot` (one cp.async group per step;
  // 16-byte pieces past L1, which keeps the tables); c: the step's cell
  auto issue = [&](int slot, int pl, long c) {
    if (col_ok && pl >= 0 && pl < NS) {
      unsigned char* dst = sm + S::o_src + (slot * arrays * G + g) * S::SRC + 16 * h;
      if (h == 0) {
        const unsigned cd = (unsigned)__cvta_generic_to_shared(sm + S::o_cls + (slot * G + g) * 4);
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(cd), "l"(a.cell_class + c) : "memory");
      }
      const size_t at = (reinterpret_cast<size_t>(src0 + c * N) & ~(size_t)15) + 16 * h;
#pragma unroll
      for (int k = 0; k < KC; ++k)
        if (S::CH % H == 0 || h + H * k < S::CH)
          cp_async_16(dst + 16 * H * k, reinterpret_cast<const void*>(at + 16 * H * k));
      if (FM >= 1 && arrays == 2) {
        const size_t ai = (reinterpret_cast<size_t>(a.iso + c * N) & ~(size_t)15) + 16 * h;
#pragma unroll
        for (int k = 0; k < KC; ++k)
          if (S::CH % H == 0 || h + H * k < S::CH)
            cp_async_16(dst + G * S::SRC + 16 * H * k, reinterpret_cast<const void*>(ai + 16 * H * k));
      }
    }
    cp_async_commit();
  };

  __syncwarp();  // the slot's last task has been read to its end
  // upwind values at the start: the boundary's, until a neighbour's or an edge's
  // (every lane writes its row's and its column's ghost cell, the lanes of one alike; the
  // barrier orders the first step's edge words after them)
  for (int i = h; i < N; i += H) {
    put(s_x, i, bS);
    put(s_gx, i, bX);
    if (DIM == 3) put(s_gy, i, bY);
  }
  __syncwarp();
#pragma unroll
  for (int j = 0; j < S::PF; ++j) issue(j, j - lx - ly, cell + j * cstep);

  // ---- the lane's rows of the face products F_a psi_up,a, as row pairs: two
  // rows of a face, or (a single row per face) one row of x and one of another face
  constexpr bool kMix = !kAdj && KF % 2 != 0;   // the last rows of x and the next axis go together
  constexpr int FP = KF / 2;                    // row pairs within a face
  constexpr int NFR = DIM * FP + (kMix ? (DIM == 2 ? 1 : 2) : 0);
  constexpr bool kFReg = NFR * FD * DB <= 192;  // kept in registers for the task
  P fr[kFReg ? NFR : 1][kFReg ? FD : 1];
  // column u of row pair n, laid out like the inverse tables (group_face_table)
  const unsigned char* face = reinterpret_cast<const unsigned char*>(a.face_group) + DB * h;
  auto face_pair = [&](int n, int u) -> P {
    const unsigned char* at = face + DB * H * (n * FD + u);
    P v;
    if constexpr (DB == 16) {
      K::from16(ldg_keep(reinterpret_cast<const uint4*>(at)), &v);
    } else {
      v = __ldg(reinterpret_cast<const f2*>(at));
    }
    return v;
  };
  if constexpr (kFReg) {
#pragma unroll
    for (int n = 0; n < NFR; ++n)
#pragma unroll
      for (int u = 0; u < FD; ++u) fr[n][u] = face_pair(n, u);
  }
  auto out_of = [](int ax, int u) { return ax == 0 ? C::x_out(u) : (ax == AS ? C::s_out(u) : C::y_out(u)); };

  const bool recv_x = col_ok && lx == 0 && tx > 0;
  const bool recv_y = DIM == 3 && col_ok && ly == 0 && ty > 0;
  const bool pub_x = col_ok && tx + 1 < a.tiles_x && lx == WX - 1;
  const bool pub_y = DIM == 3 && col_ok && ty + 1 < a.tiles_y && ly == WY - 1;
  // edge words of plane 0 (from one plane to the next: WY or WX times FD * W)
  constexpr long EX = (long)WY * FD * W, EY = (long)WX * FD * W;
  const unsigned long long* in_x = a.edge_x + (((size_t)d * tiles + tile - 1) * NS * WY + ly) * (FD * W) + h;
  const unsigned long long* in_y = a.edge_y + (((size_t)d * tiles + tile - a.tiles_x) * NS * WX + lx) * (FD * W) + h;
  unsigned long long* out_x = a.edge_x + (((size_t)d * tiles + tile) * NS * WY + ly) * (FD * W) + h;
  unsigned long long* out_y = a.edge_y + (((size_t)d * tiles + tile) * NS * WX + lx) * (FD * W) + h;
  unsigned long long rX[KE], rY[DIM == 3 ? KE : 1];
  bool hX = false, hY = false;

  // the lane's rows of the inverse stay in registers while its column's material
  // does not change, where they take at most 64 registers
  constexpr int PJ = 16 / DB, PL = 16 / SZ;  // columns per 16-byte piece of a row pair, of the lone row
  constexpr int NCP = RW::pair_pieces(SZ), NCL = RW::lone_pieces(SZ);
  constexpr bool kCache = R * N * SZ <= 256;
  P tab[kCache && RP ? RP : 1][kCache ? NCP * PJ : 1];
  real tlone[kCache && kOdd ? N : 1];
  const unsigned char* cached = nullptr;

  const int nsteps = NS + WX - 1 + WY - 1;
  int slot = 0, fill = S::PF;
  for (int s = 0; s < nsteps; ++s, cell += cstep) {
    const int sc = s - lx - ly;
    const bool act = col_ok && sc >= 0 && sc < NS;
    // ---- upwind tile's outflow into the ghost cells
    bool failed = false;
    const unsigned tag = want_epoch | ((unsigned)sc & 0xffffu);
    if (act && recv_x) {
#pragma unroll
      for (int k = 0; k < KE; ++k) {
        const int w = h + H * k;
        if ((FD * W) % H == 0 || w < FD * W) {
          unsigned v = (unsigned)rX[k];
          if (!(hX && (unsigned)(rX[k] >> 32) == tag))
            failed |= !poll_word(in_x + sc * EX + H * k, tag, &v, a.status, a.wait_limit_ns);
          reinterpret_cast<unsigned*>(s_gx)[C::x_out(w / W) * W + w % W] = v;
        }
      }
    }
    if (DIM == 3 && act && recv_y) {
#pragma unroll
      for (int k = 0; k < KE; ++k) {
        const int w = h + H * k;
        if ((FD * W) % H == 0 || w < FD * W) {
          unsigned v = (unsigned)rY[k];
          if (!(hY && (unsigned)(rY[k] >> 32) == tag))
            failed |= !poll_word(in_y + sc * EY + H * k, tag, &v, a.status, a.wait_limit_ns);
          reinterpret_cast<unsigned*>(s_gy)[C::y_out(w / W) * W + w % W] = v;
        }
      }
    }
    if (__any_sync(FULL, failed)) {  // status is set; drain own copies, leave
      cp_async_wait<0>();
      break;
    }
    // the next plane's words, one step ahead (tags are checked when used)
    hX = recv_x && sc + 1 >= 0 && sc + 1 < NS;
    if (hX) {
#pragma unroll
      for (int k = 0; k < KE; ++k)
        if ((FD * W) % H == 0 || h + H * k < FD * W) rX[k] = ld_relaxed_u64(in_x + (sc + 1) * EX + H * k);
    }
    hY = recv_y && sc + 1 >= 0 && sc + 1 < NS;
    if (DIM == 3 && hY) {
#pragma unroll
      for (int k = 0; k < KE; ++k)
        if ((FD * W) % H == 0 || h + H * k < FD * W) rY[k] = ld_relaxed_u64(in_y + (sc + 1) * EY + H * k);
    }
    __syncwarp();
    // ---- face products
    if (act) {
#pragma unroll
      for (int ax = 0; ax < DIM; ++ax) {
        if (FP == 0) break;
        const unsigned char* from = ax == 0 ? up_x : (ax == AS ? s_x : up_y);
        typename K::Acc acc[FP ? FP : 1];
        real upv[FD];
        if (kAdj && ax > 0) {  // neighbours along x: 16 bytes (FP32: 8) at a time
#pragma unroll
          for (int u = 0; u < FD; u += 2) {
            const P v = K::array_load(from + out_of(ax, u) * SZ);
            upv[u] = K::get(v, 0);
            upv[u + 1 < FD ? u + 1 : u] = K::get(v, 1);
          }
        } else {
#pragma unroll
          for (int u = 0; u < FD; ++u) upv[u] = get(from, out_of(ax, u));
        }
#pragma unroll
        for (int u = 0; u < FD; ++u) {
          const typename K::Op up = K::op(K::make(upv[u], upv[u]));
#pragma unroll
          for (int k = 0; k < FP; ++k) {
            const P row = kFReg ? fr[kFReg ? ax * FP + k : 0][kFReg ? u : 0] : face_pair(ax * FP + k, u);
            if (u == 0) acc[k] = K::prod(row, up, z);
            else K::fma(acc[k], row, up, z);
          }
        }
#pragma unroll
        for (int k = 0; k < FP; ++k) {
          const P v = K::raw(acc[k]);
          if constexpr (kAdj) {
            const int m = h + H * k;
            if ((FD / 2) % H == 0 || m < FD / 2) K::store(s_f + (ax * (FD / 2) + m) * DB, v);
          } else {
            const int t0 = h + H * (2 * k), t1 = t0 + H;
            put(s_f, ax * FD + t0, K::get(v, 0));
            if (FD % H == 0 || t1 < FD) put(s_f, ax * FD + t1, K::get(v, 1));
          }
        }
      }
      if constexpr (kMix) {
        const int t = h + H * (KF - 1);
        typename K::Acc acc{};
#pragma unroll
        for (int u = 0; u < FD; ++u) {
          const P row = kFReg ? fr[kFReg ? DIM * FP : 0][kFReg ? u : 0] : face_pair(DIM * FP, u);
          const typename K::Op up = K::op(
              K::make(get(up_x, C::x_out(u)), DIM == 2 ? get(s_x, C::s_out(u)) : get(up_y, C::y_out(u))));
          if (u == 0) acc = K::prod(row, up, z);
          else K::fma(acc, row, up, z);
        }
        const P v = K::raw(acc);
        if (FD % H == 0 || t < FD) {
          put(s_f, t, K::get(v, 0));
          put(s_f, FD + t, K::get(v, 1));
        }
        if constexpr (DIM == 3) {  // the sweep-axis row alone
          typename A::acc as = A::zero();
#pragma unroll
          for (int u = 0; u < FD; ++u) {
            const real row = K::get(kFReg ? fr[kFReg ? DIM * FP + 1 : 0][kFReg ? u : 0] : face_pair(DIM * FP + 1, u), 0);
            const real up = get(s_x, C::s_out(u));
            if (u == 0) as = A::prod(row, up);
            else A::fma(as, row, up);
          }
          if (FD % H == 0 || t < FD) put(s_f, 2 * FD + t, A::raw(as));
        }
      }
    }
    cp_async_wait<S::PF - 1>();  // this step's source has landed
    __syncwarp();
    // ---- right-hand side, into the cell's slot (its psi has been read)
    const unsigned char* Ai = ainv;
    if (act) {
      const unsigned char* src = sm + S::o_src + (slot * arrays * G + g) * S::SRC;
      const unsigned char* isrc = src + G * S::SRC;
      Ai += reinterpret_cast<const int*>(sm + S::o_cls)[slot * G + g] * ainv_class;
      if constexpr (kAdj) {  // (a cell's bytes are a multiple of 16: no offset)
        // value t of the x face, stored in pairs
        auto pair_half = [&](int t) {
          const unsigned char* q = s_f + (t / 2) * DB;
          if constexpr (std::is_same<real, df64>::value)
            return df64(reinterpret_cast<const float*>(q)[t % 2], reinterpret_cast<const float*>(q)[2 + t % 2]);
          else
            return get(q, t % 2);
        };
#pragma unroll
        for (int p = 0; p < RP; ++p) {
          const int m = h + H * p, i = 2 * m;
          if ((N / 2) % H == 0 || m < N / 2) {
            P v = K::swap_if(K::array_load(src + po[p] * SZ), swap);
            if (FM >= 1) {
              typename K::Acc acc = K::from(arrays == 2 ? K::swap_if(K::array_load(isrc + po[p] * SZ), swap)
                                                        : K::make(real(0), real(0)));
              K::fma(acc, K::make(w0, w0), K::op(v), z);
              v = K::raw(acc);
            }
            bool on[3] = {false, false, false};  // some lane's pair lies on the inflow face of the axis
#pragma unroll
            for (int l = 0; l < H; ++l)
#pragma unroll
              for (int ax = 0; ax < DIM; ++ax)
                if (l + H * p < N / 2 && C::comp(2 * (l + H * p), ax) == 0) on[ax] = true;
            if (on[0] && C::comp(i, 0) == 0) {  // the pair's first dof
              typename A::acc acc = A::from(K::get(v, 0));
              A::fma(acc, wX, pair_half(i / P1));
              v = K::make(A::raw(acc), K::get(v, 1));
            }
            if (on[AS] && C::comp(i, AS) == 0) {
              typename K::Acc acc = K::from(v);
              K::fma(acc, K::make(wS, wS), K::op(K::load(s_f + (AS * (FD / 2) + m) * DB)), z);
              v = K::raw(acc);
            }
            if (DIM == 3 && on[1] && C::comp(i, 1) == 0) {
              typename K::Acc acc = K::from(v);
              K::fma(acc, K::make(wY, wY), K::op(K::load(s_f + (FD / 2 + (i % P1 + P1 * (i / (P1 * P1))) / 2) * DB)), z);
              v = K::raw(acc);
            }
            K::array_put(s_x + i * SZ, v);
          }
        }
      } else {
        const int o0 = S::GR == 16 ? 0 : (int)(reinterpret_cast<size_t>(src0 + cell * N) & 15);
        const int o1 = FM == 0 || S::GR == 16 ? 0 : (int)(reinterpret_cast<size_t>(a.iso + cell * N) & 15);
#pragma unroll
        for (int k = 0; k < R; ++k) {
          const int i = h + H * k;
          if (N % H == 0 || i < N) {
            real v = *reinterpret_cast<const real*>(src + o0 + po[k] * SZ);
            if (FM >= 1) {
              typename A::acc acc =
                  A::from(arrays == 2 ? *reinterpret_cast<const real*>(isrc + o1 + po[k] * SZ) : real(0));
              A::fma(acc, w0, v);
              v = A::raw(acc);
            }
            bool on[3] = {false, false, false};
#pragma unroll
            for (int l = 0; l < H; ++l)
#pragma unroll
              for (int ax = 0; ax < DIM; ++ax)
                if (l + H * k < N && C::comp(l + H * k, ax) == 0) on[ax] = true;
            auto term = [&](real w, int f) {
              typename A::acc acc = A::from(v);
              A::fma(acc, w, get(s_f, f));
              v = A::raw(acc);
            };
            if (on[0] && C::comp(i, 0) == 0) term(wX, i / P1);
            if (on[AS] && C::comp(i, AS) == 0) term(wS, AS * FD + i);
            if (DIM == 3 && on[1] && C::comp(i, 1) == 0) term(wY, FD + i % P1 + P1 * (i / (P1 * P1)));
            put(s_x, i, v);
          }
        }
      }
    }
    issue(fill, sc + S::PF, cell + S::PF * cstep);  // refills the slot consumed a step ago
    slot = slot + 1 == S::RING ? 0 : slot + 1;
    fill = fill + 1 == S::RING ? 0 : fill + 1;
    __syncwarp();
    // ---- x = A'^-1 b, this lane's rows
    P xp2[RP ? RP : 1];
    real xl = real(0);
    if (act) {
      typename K::Acc acc[RP ? RP : 1];
      typename A::acc al = A::zero();
      if constexpr (kCache) {
        if (Ai != cached) {  // another material: its rows replace the ones in registers
          cached = Ai;
#pragma unroll
          for (int c = 0; c < NCP; ++c)
#pragma unroll
            for (int p = 0; p < RP; ++p)
              K::from16(ldg_keep(reinterpret_cast<const uint4*>(Ai + 16 * H * (p * NCP + c))), &tab[p][c * PJ]);
          if constexpr (kOdd)
#pragma unroll
            for (int c = 0; c < NCL; ++c) {
              real l[PL];
              load_row<real, PL>(reinterpret_cast<const real*>(Ai + 16 * H * (RP * NCP + c)), l);
#pragma unroll
              for (int j = 0; j < PL; ++j)
                if (c * PL + j < N) tlone[c * PL + j] = l[j];
            }
        }
      }
      constexpr int NB = (N + PL - 1) / PL;  // 16-byte pieces of b
      // the loop over b whole in the code while it stays within some 1500 packed
      // operations (its table loads then run ahead: 3-D Q3 double-float 7.47 ms
      // against 9.05 two pieces at a time, 32^3 LS S8), else two pieces at a time
      // (past the instruction cache: 3-D Q5 2.14 ms whole, 0.97 two at a time, 8^3)
      constexpr int kOps = std::is_same<real, df64>::value ? 10 : (SZ == 8 ? 2 : 1);
      constexpr int U = (RP + (kOdd ? 1 : 0)) * kOps * N <= 1300 ? NB : 2;
      auto piece = [&](int c, bool first) {
        real bv[PL];
        load_row_shared<real, PL>(s_x + 16 * c, bv);
        typename K::Op bo[PL];
#pragma unroll
        for (int j = 0; j < PL; ++j) bo[j] = K::op(K::make(bv[j], bv[j]));
        real l[PL];
        if (kOdd && !kCache)
          load_row<real, PL>(reinterpret_cast<const real*>(Ai + 16 * H * (RP * NCP + c)), l);
#pragma unroll
        for (int j0 = 0; j0 < PL; j0 += PJ) {
          if (N % PL != 0 && c * PL + j0 >= N) break;
#pragma unroll
          for (int p = 0; p < RP; ++p) {
            P row[PJ];
            if constexpr (!kCache)
              K::from16(ldg_keep(reinterpret_cast<const uint4*>(Ai + 16 * H * (p * NCP + c * (PL / PJ) + j0 / PJ))), row);
#pragma unroll
            for (int j = 0; j < PJ; ++j) {
              const int col = c * PL + j0 + j;
              if (N % PL != 0 && col >= N) break;
              const P rv = kCache ? tab[kCache ? p : 0][kCache ? col : 0] : row[j];
              if (first && j0 + j == 0) acc[p] = K::prod(rv, bo[j0 + j], z);
              else K::fma(acc[p], rv, bo[j0 + j], z);
            }
          }
        }
        if constexpr (kOdd) {
#pragma unroll
          for (int j = 0; j < PL; ++j) {
            const int col = c * PL + j;
            if (N % PL != 0 && col >= N) break;
            const real rv = kCache ? tlone[kCache ? col : 0] : l[j];
            if (first && j == 0) al = A::prod(rv, bv[0]);
            else A::fma(al, rv, bv[j]);
          }
        }
      };
      piece(0, true);
#pragma unroll U
      for (int c = 1; c < NB; ++c) piece(c, false);
#pragma unroll
      for (int p = 0; p < RP; ++p) xp2[p] = K::result(acc[p]);
      if (kOdd) xl = A::get(al);
    }
    __syncwarp();  // every lane has read b
    if (act) {
      if constexpr (kAdj) {
#pragma unroll
        for (int p = 0; p < RP; ++p)
          if ((N / 2) % H == 0 || h + H * p < N / 2) K::array_put(s_x + 2 * (h + H * p) * SZ, xp2[p]);
      } else {
#pragma unroll
        for (int k = 0; k < R; ++k)
          if (N % H == 0 || h + H * k < N)
            put(s_x, h + H * k, k / 2 < RP ? K::get(xp2[k / 2 < RP ? k / 2 : 0], k % 2) : xl);
      }
    }
    __syncwarp();
    // ---- outflow of the tile's last cells first (the downwind tiles wait on it), then psi
    if (act) {
      const unsigned long long ptag = (unsigned long long)((a.epoch << 16) | ((unsigned)sc & 0xffffu)) << 32;
      if (pub_x) {
#pragma unroll
        for (int k = 0; k < KE; ++k) {
          const int w = h + H * k;
          if ((FD * W) % H == 0 || w < FD * W)
            st_relaxed_u64(out_x + sc * EX + H * k, ptag | reinterpret_cast<const unsigned*>(s_x)[C::x_out(w / W) * W + w % W]);
        }
      }
      if (pub_y) {
#pragma unroll
        for (int k = 0; k < KE; ++k) {
          const int w = h + H * k;
          if ((FD * W) % H == 0 || w < FD * W)
            st_relaxed_u64(out_y + sc * EY + H * k, ptag | reinterpret_cast<const unsigned*>(s_x)[C::y_out(w / W) * W + w % W]);
        }
      }
      real* out = a.psi + dirbase + cell * N;
#pragma unroll
      for (int k = 0; k < (kAdj ? RP : R); ++k) {
        if constexpr (kAdj) {
          if ((N / 2) % H == 0 || h + H * k < N / 2) K::array_store(out + po[k], K::swap_if(xp2[k], swap));
        } else {
          if (N % H == 0 || h + H * k < N)
            store_stream(out + po[k], k / 2 < RP ? K::get(xp2[k / 2 < RP ? k / 2 : 0], k % 2) : xl);
        }
      }
    }
  }
}

// Resident blocks per SM the registers are cut for (0: the compiler's choice).  Left to
// itself the compiler settled on anything between 64 and 168 registers, another number
// after every change around the loops, and the loads of the tables run ahead as far as
// there are registers: with three blocks they do.  Sweep kernel, double-float / FP32,
// us, the compiler's choice -> 3 blocks (4 in FP32 up to 16 dofs):
//   2-D Q3 135x93 LS S12  466 / 235 -> 446 / 223    2-D Q4 100^2 S8, 16 materials  954 / 346 -> 653 / 264
//   2-D Q5 64^2 LS S8, 16 materials  731 / 252 -> 488 / 192
//   3-D Q2 24^3 LS S6     636 / 243 -> 581 / 238    3-D Q3 16^3 S4, 16 materials   956 / 247 -> 556 / 169
//   3-D Q4 10^3 LS S4     522 / 163 -> 491 / 110    3-D Q5 8^3 S4                  837 / 536 -> 735 / 227
// (five blocks: 3-D Q5 2345 / 424; FP32 3-D Q2 48^3 S8 with 8 lanes is the one exception,
// 2233 -> 2390).
template <typename real, int DIM, int P1, int H>
constexpr int group_blocks() {
  constexpr int N = Cell<DIM, P1>::N;
  if (sizeof(real) == 4 && N == 27 && H == 8) return 0;
  return sizeof(real) == 4 && N <= 16 ? 4 : 3;
}
template <typename real, int DIM, int P1, int FM, int H>
__global__ void __launch_bounds__(128, (group_blocks<real, DIM, P1, H>())) sweep_group_kernel(const __grid_constant__ SweepArgs<real> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr unsigned FULL = 0xffffffffu;
  // With queues, an SM starts on one |Omega| class, whose tables its L1 then holds, and
  // goes on to the next when that has no tasks left.  Every queue is in dependency
  // order and a class's tasks wait on none of another's, so any warp may take the
  // head of any queue.
  int queue = 0;
  if (a.n_queues > 1) {
    unsigned sm;
    asm("mov.u32 %0, %%smid;" : "=r"(sm));
    queue = (int)(sm % (unsigned)a.n_queues);
  }
  for (;;) {
    int task = 0, stop = 0;
    if ((threadIdx.x & 31) == 0) {
      task = atomicAdd(a.ticket + queue, 1);
      stop = *(volatile int*)a.status;
    }
    task = __shfl_sync(FULL, task, 0);
    stop = __shfl_sync(FULL, stop, 0);
    if (stop) return;
    int count = a.n_tasks;
    if (a.n_queues > 1) {
      const int first = a.queue_first[queue];
      count = a.queue_first[queue + 1];
      task += first;
    }
    if (task >= count) {
      if (a.n_queues <= 1) return;
      // the next queue with tasks left, from all counters at once (asking one after the
      // other cost an atomic each, of every idle warp: 2-D Q3 64^2 LS S16 FP32, 36
      // queues, 233 us where one queue takes 125)
      const int lane = threadIdx.x & 31;
      unsigned long long open = 0;
#pragma unroll
      for (int part = 0; part < 2; ++part) {
        const int k = 32 * part + lane;
        const bool some = k < a.n_queues && *(volatile int*)(a.ticket + k) < a.queue_first[k + 1] - a.queue_first[k];
        open |= (unsigned long long)__ballot_sync(FULL, some) << 32 * part;
      }
      if (!open) return;
      const unsigned long long after = open >> queue >> 1 << 1 << queue;
      queue = __ffsll((long long)(after ? after : open)) - 1;
      continue;
    }
    sweep_group_task<real, DIM, P1, FM, H>(a, task, smem_raw);
  }
}

// What a batched launch of a form needs: every problem's arguments, the ticket
// map, and whether the problems bring a fixed source
template <typename real>
struct BatchLaunch {
  const SweepArgs<real>* args;
  const int2* tmap;
  int n_total;
  int* ticket;
  const int* status;
  const unsigned* epoch;
  bool sources;
  int grid, block;
};

// Many problems in one persistent launch (see sweep_batch_kernel)
template <typename real, int DIM, int P1, int FM, int H>
__global__ void __launch_bounds__(128, (group_blocks<real, DIM, P1, H>())) sweep_group_batch_kernel(const SweepArgs<real>* __restrict__ args,
                                                                const int2* __restrict__ tmap, int n_total, int* ticket,
                                                                const int* status, const unsigned* epoch) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ SweepArgs<real> s_args[4];
  for (;;) {
    const int p = next_batch_task(args, tmap, n_total, ticket, status, epoch, s_args[threadIdx.x >> 5]);
    if (p < 0) return;
    sweep_group_task<real, DIM, P1, FM, H>(s_args[threadIdx.x >> 5], p, smem_raw);
    __syncwarp();  // the slot is rewritten by the next task
  }
}

// L1 kept beside the resident blocks, for the inverse tables of the running
// directions: the sources stream past it (16-byte cp.async.cg), and 28, 64 and
// 112 KB measured the same within the spread; more where an SM's warps share one
// class's tables
constexpr int kGroupKeepKb = 64, kQueueKeepKb = 132;

template <typename real, int DIM, int P1, int FM, int H>
cudaError_t launch_group_fm(const SweepArgs<real>& a, int grid, int block, cudaStream_t s) {
  using S = GroupSlot<real, DIM, P1, H>;
  const int arrays = FM >= 1 && a.iso ? 2 : 1;
  const size_t warps = block / 32, smem = warps * S::bytes(arrays);
  static SweepLaunch st;
  const cudaError_t e = st.prepare((const void*)sweep_group_kernel<real, DIM, P1, FM, H>, arrays, grid, block, smem,
                                   warps * S::bytes(FM >= 1 ? 2 : 1), 0, a.n_queues > 1 ? kQueueKeepKb : kGroupKeepKb);
  if (e != cudaSuccess) return e;
  sweep_group_kernel<real, DIM, P1, FM, H><<<grid, block, smem, s>>>(a);
  return cudaGetLastError();
}
template <typename real, int DIM, int P1, int FM, int H>
cudaError_t launch_group_batch_fm(const BatchLaunch<real>& b, cudaStream_t s) {
  using S = GroupSlot<real, DIM, P1, H>;
  const int arrays = FM >= 1 && b.sources ? 2 : 1;
  const size_t warps = b.block / 32, smem = warps * S::bytes(arrays);
  static SweepLaunch st;
  const cudaError_t e = st.prepare((const void*)sweep_group_batch_kernel<real, DIM, P1, FM, H>, arrays, b.grid, b.block, smem,
                                   warps * S::bytes(FM >= 1 ? 2 : 1), 4 * sizeof(SweepArgs<real>), kGroupKeepKb);
  if (e != cudaSuccess) return e;
  sweep_group_batch_kernel<real, DIM, P1, FM, H>
      <<<b.grid, b.block, smem, s>>>(b.args, b.tmap, b.n_total, b.ticket, b.status, b.epoch);
  return cudaGetLastError();
}

// The forms that are instantiated (default_lanes in operator.cu picks among them);
// a fused moment where the cell has at most 16 dofs
#define OURANOS_GROUP_FORMS(CASE)                                        \
  if constexpr (DIM == 2) {                                              \
    CASE(3, 4) CASE(4, 2) CASE(4, 8) CASE(5, 2) CASE(5, 8) CASE(6, 16)   \
  } else {                                                               \
    CASE(3, 2) CASE(3, 8) CASE(3, 16) CASE(4, 16) CASE(5, 32) CASE(6, 32) \
  }

template <typename real, int DIM>
cudaError_t launch_group_dim(int p1, int fm, const SweepArgs<real>& a, int grid, int block, cudaStream_t s) {
#define CASE(P, HH)                                                                              \
  if (p1 == P && a.lpc == HH) {                                                                  \
    if (fm == 0) return launch_group_fm<real, DIM, P, 0, HH>(a, grid, block, s);                 \
    if constexpr (Cell<DIM, P>::N <= 16)                                                         \
      if (fm == 1) return launch_group_fm<real, DIM, P, 1, HH>(a, grid, block, s);               \
  }
  OURANOS_GROUP_FORMS(CASE)
#undef CASE
  return cudaErrorInvalidValue;
}
template <typename real, int DIM>
cudaError_t launch_group_batch_dim(int p1, int fm, int lpc, const BatchLaunch<real>& b, cudaStream_t s) {
#define CASE(P, HH)                                                                              \
  if constexpr (P <= (DIM == 2 ? 5 : 3))                                                         \
    if (p1 == P && lpc == HH) {                                                                  \
      if (fm == 0) return launch_group_batch_fm<real, DIM, P, 0, HH>(b, s);                      \
      if constexpr (Cell<DIM, P>::N <= 16)                                                       \
        if (fm == 1) return launch_group_batch_fm<real, DIM, P, 1, HH>(b, s);                    \
    }
  OURANOS_GROUP_FORMS(CASE)
#undef CASE
  return cudaErrorInvalidValue;
}

}  // namespace ouranos
