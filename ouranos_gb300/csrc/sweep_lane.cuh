// The sweep with one lane to a cell for cells of at most nine dofs (2-D Q1 and
// Q2, 3-D Q1), the default form where a problem has warps enough: a task is one
// direction crossing a tile of 32 cells (2-D 32 x 1, 3-D 4 x 8), lane (lx, ly)
// working on plane s - lx - ly at step s as in sweep.cuh, whose orientation,
// tickets, edge words and bounded waits are used unchanged.
//
// What bounds it is the issue slots of a step and the 128 bytes a clock of the
// L1 / shared-memory pipe, so:
//   - rows of the cell solve, of the face products and the face terms go two at a
//     time in packed FP32 operations (pack2.cuh);
//   - whatever touches memory does so for the whole warp at once: the lanes copy
//     the 32 cells' sources piece by piece (neighbouring lanes, neighbouring 16
//     bytes) into a shared ring, and psi and the edge words leave through a
//     shared slot the same way; a lane copying its own cell met 32 lines per
//     instruction, one clock each;
//   - in FP32 the 32 bytes of a 3-D Q1 cell leave their lane in one store, 32 clocks
//     of that pipe (through the slot 56: two-way conflicts going in, the read, two
//     stores of 16 lines), and its source is read 16 bytes at a time: sweep kernel of
//     128^3 LS S8 4604 -> 4100 us.  In 2-D the cells of 32 (FP64) and 16 bytes
//     measured the same within 4 % either way and take the slot;
//   - the face mass matrices are kernel arguments (constant memory);
//   - a column's materials come four planes to a word.
// Every dof is rounded in the order of the other forms, so all give the same bits.
#pragma once

#include "sweep_group.cuh"

namespace ouranos {

// Layout of one warp's shared-memory slot (bytes)
template <typename real, int DIM, int P1>
struct LaneSlot {
  using C = Cell<DIM, P1>;
  static constexpr int N = C::N, FD = C::FD, SZ = (int)sizeof(real);
  static constexpr int CELLB = N * SZ;
  static constexpr int GR = (CELLB & -CELLB) < 16 ? (CELLB & -CELLB) : 16;
  static constexpr int CH = (CELLB + 16 - GR + 15) / 16;  // aligned 16-byte pieces that cover a cell's source
  static_assert(16 * CH - CELLB <= (int)kSrcSlack, "the sources' buffers hold the last piece");
  static constexpr int SRC = 16 * (CH | 1);               // (odd multiples of 16 bytes: different banks)
  // psi's slot: Q1 cells padded likewise; 9 values at their own stride, which meets
  // every bank once and makes the slot one array of the tile's values
  static constexpr int OUT = GR == 16 ? 16 * ((CELLB / 16) | 1) : CELLB;
  static constexpr int PF = 2, RING = PF + 1;             // planes in flight ahead of the one being solved
  static constexpr int WX = DIM == 2 ? 32 : 4, WY = 32 / WX;
  static constexpr int EB = (FD * SZ + 15) / 16 * 16;     // an edge's face values
  // one store per cell: the slot holds the outflow edges only
  static constexpr bool kDirect = DIM == 3 && P1 == 2 && SZ == 4;
  static constexpr int o_ox = 0, o_oy = WY * EB;
  static constexpr int o_ex = kDirect ? (WY + WX) * EB : 32 * OUT;
  static constexpr int o_ey = o_ex + WY * EB;
  static constexpr int o_cls = o_ey + (DIM == 3 ? WX * EB : 0);
  static constexpr int CW = 4;                            // class words in flight per column
  static constexpr int o_src = o_cls + CW * 128;
  __host__ __device__ static constexpr int bytes(int arrays) { return o_src + RING * arrays * 32 * SRC; }
};

// ldg_keep in program order: the loads stay ahead of the arithmetic that follows
__device__ __forceinline__ uint4 ldg_first(const unsigned char* p) {
  uint4 u;
  asm volatile("ld.global.nc.L1::evict_last.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(u.x), "=r"(u.y), "=r"(u.z), "=r"(u.w)
               : "l"(p));
  return u;
}

// FD values of an edge slot: 16 bytes a load, or one value where registers are short
template <bool VEC, int FD, typename real, int NV>
__device__ __forceinline__ void load_edge(real (&v)[NV], const unsigned char* from) {
  if constexpr (VEC) {
#pragma unroll
    for (int k = 0; k < NV * (int)sizeof(real) / 16; ++k) {
      const uint4 u = *reinterpret_cast<const uint4*>(from + 16 * k);
      memcpy(v + k * (16 / sizeof(real)), &u, 16);
    }
  } else {
#pragma unroll
    for (int t = 0; t < FD; ++t) v[t] = *reinterpret_cast<const real*>(from + t * sizeof(real));
  }
}

// the pairs of a Q1 cell between canonical and physical order: pair m of the one is
// pair m ^ flips of the other, its values swapped where x is flipped
__device__ __forceinline__ void flip_pairs(f2 (&v)[4], int flip) {
#pragma unroll
  for (int m = 0; m < 4; ++m) v[m] = Pk<float>::swap_if(v[m], flip & 1);
#pragma unroll
  for (int ax = 1; ax < 3; ++ax) {
    const bool f = flip & (1 << ax);
#pragma unroll
    for (int m = 0; m < 4; ++m)
      if (!(m & ax)) {
        const f2 lo = v[m], hi = v[m | ax];
        v[m] = f ? hi : lo;
        v[m | ax] = f ? lo : hi;
      }
  }
}
// eight FP32 values in one streaming store of 32 bytes
__device__ __forceinline__ void store_cell(void* to, const f2 (&v)[4]) {
  asm volatile("st.global.cs.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(to), "f"(f2_get(v[0], 0)),
               "f"(f2_get(v[0], 1)), "f"(f2_get(v[1], 0)), "f"(f2_get(v[1], 1)), "f"(f2_get(v[2], 0)),
               "f"(f2_get(v[2], 1)), "f"(f2_get(v[3], 0)), "f"(f2_get(v[3], 1))
               : "memory");
}

template <typename real, int DIM, int P1, int FM>
__device__ __forceinline__ void sweep_lane_task(const SweepArgs<real>& a, const int task, unsigned char* smem_raw) {
  using S = LaneSlot<real, DIM, P1>;
  using RW = GroupRows<DIM, P1, 1>;
  using C = Cell<DIM, P1>;
  using A = Arith<real>;
  using K = Pk<real>;
  using P = typename K::P;
  constexpr int N = S::N, FD = S::FD, SZ = S::SZ, CH = S::CH, WX = S::WX, WY = S::WY;
  constexpr int RP = RW::RP;
  constexpr bool kOdd = RW::kOdd;
  constexpr bool kAligned = S::GR == 16;
  constexpr int W = Tagged<real>::W;
  constexpr int AS = DIM - 1;
  constexpr unsigned FULL = 0xffffffffu;
  // edge words: of the x edge (WY cells) and, in 3-D, of the y edge (WX cells)
  constexpr int FW = FD * W;
  constexpr int NEX = (WY * FW + 31) / 32, NEY = DIM == 3 ? (WX * FW + 31) / 32 : 0;
  const int lane = threadIdx.x & 31;
  const int lx = lane % WX, ly = lane / WX;
  const int arrays = FM == 0 ? 1 : (a.iso ? 2 : 1);
  unsigned char* sm = smem_raw + (threadIdx.x >> 5) * S::bytes(arrays);
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
  auto phys = [&](int i) {
    return base + C::comp(i, 0) * st0 + C::comp(i, 1) * st1 + (DIM == 3 ? C::comp(i, 2) * st2 : 0);
  };
  const bool swap = flip & 1;  // Q1: the two dofs of an x pair change places
  const int sflip = DIM == 3 ? (flip & 4) : (flip & 2);
  const int plane = DIM == 2 ? NX : NX * NY;     // (cell numbers fit an int)
  const int cstep = sflip ? -plane : plane;      // cells from one step to the next
  const int cell0 = sflip ? plane * (NS - 1) : 0;
  // column (xc, yc) of the canonical tile: its cell at step 0, walking in from
  // outside the mesh (used on the column's planes only)
  auto cell_of_group = [&](int g) {
    const int gx = tx * WX + g % WX, gy = ty * WY + g / WX;
    const int xp = (flip & 1) ? NX - 1 - gx : gx;
    const int yp = DIM == 3 ? ((flip & 2) ? NY - 1 - gy : gy) : 0;
    return cell0 + xp + NX * yp - cstep * (g % WX + g / WX);
  };
  const int xc = tx * WX + lx, yc = ty * WY + ly;
  const bool col_ok = xc < NX && (DIM == 2 || yc < NY);
  const int skew = lx + ly;
  const size_t dirbase = (size_t)d * a.n_dofs;
  const unsigned char* ainv = reinterpret_cast<const unsigned char*>(a.ainv) +
                              (size_t)a.dir_class[d] * RW::matrix_bytes(SZ);
  const unsigned ainv_class = (unsigned)a.n_dir_class * RW::matrix_bytes(SZ);
  const unsigned char* src0 = reinterpret_cast<const unsigned char*>(FM == 0 ? a.q + dirbase : a.src);

  // piece j of the source copies: cell (lane + 32 j) / CH of the tile
  int sc_cell[CH];
#pragma unroll
  for (int j = 0; j < CH; ++j) sc_cell[j] = cell_of_group((lane + 32 * j) / CH);
  auto active = [&](int s) {  // the tile's cells with a plane at step s
    return __ballot_sync(FULL, col_ok && (unsigned)(s - skew) < (unsigned)NS);
  };
  // materials of the lane's column, in words of four planes (a byte each) or, with
  // more than 256 classes, of one plane; words go through a shared ring
  const int ncol = plane;
  const int col = cell_of_group(lane) + cstep * skew - cell0;  // physical column
  const bool bytes = a.cls4 != nullptr;
  const unsigned* cls4 = a.cls4 + (sflip ? (size_t)ncol * ((NS + 3) / 4) : 0) + col;
  auto class_word = [&](int w) {  // word w of the column into its slot
    const int pl = bytes ? 4 * w : w;
    if (col_ok && pl >= 0 && pl < NS) {
      const void* from = bytes ? (const void*)(cls4 + (size_t)w * ncol)
                               : (const void*)(a.cell_class + col + (long)plane * (sflip ? NS - 1 - w : w));
      const unsigned to = (unsigned)__cvta_generic_to_shared(sm + S::o_cls + (w & (S::CW - 1)) * 128 + lane * 4);
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(to), "l"(from) : "memory");
    }
  };
  // the sources of step s into ring slot `slot` (one cp.async group per step;
  // 16-byte pieces past L1, which keeps the tables)
  auto issue = [&](int slot, int s, unsigned on) {
    const int adv = s * cstep;
    unsigned char* to = sm + S::o_src + slot * arrays * 32 * S::SRC;
    auto piece = [&](int j) {
      const int u = lane + 32 * j, g = u / CH, p = u - g * CH;
      const long cb = (long)(sc_cell[j] + adv) * S::CELLB;
      unsigned char* dst = to + g * S::SRC + 16 * p;
      size_t at = reinterpret_cast<size_t>(src0) + cb;
      if (!kAligned) at &= ~(size_t)15;
      cp_async_16(dst, reinterpret_cast<const void*>(at + 16 * p));
      if (FM >= 1 && arrays == 2) {
        size_t ai = reinterpret_cast<size_t>(a.iso) + cb;
        if (!kAligned) ai &= ~(size_t)15;
        cp_async_16(dst + 32 * S::SRC, reinterpret_cast<const void*>(ai + 16 * p));
      }
    };
    if (on == FULL) {
#pragma unroll
      for (int j = 0; j < CH; ++j) piece(j);
    } else {
#pragma unroll
      for (int j = 0; j < CH; ++j)
        if ((on >> ((lane + 32 * j) / CH)) & 1u) piece(j);
    }
  };

  __syncwarp();  // the slot's last task has been read to its end
  // The inflow, until an edge brings a neighbour's values: every lane writes it to its
  // row's and its column's slot (the same value from all lanes of one).  The edge words
  // of the first step are written by other lanes than these: the barrier orders the two.
  for (int t = 0; t < FD; ++t) {
    *reinterpret_cast<real*>(sm + S::o_ex + ly * S::EB + t * SZ) = bX;
    if (DIM == 3) *reinterpret_cast<real*>(sm + S::o_ey + lx * S::EB + t * SZ) = bY;
  }
  __syncwarp();
  class_word(0);
  class_word(1);
#pragma unroll
  for (int j = 0; j < S::PF; ++j) {
    issue(j, j, active(j));
    cp_async_commit();
  }
  // psi, 9-dof cells: value lane + 32 j of the tile, in values from the step's cell
  constexpr int NP = kAligned ? 1 : N;
  int po[NP];
  if (!kAligned) {
#pragma unroll
    for (int j = 0; j < NP; ++j) {
      const int u = lane + 32 * j, g = u / N;
      po[j] = cell_of_group(g) * N + (u - g * N);
    }
  }

  real psiX[FD], psiY[DIM == 3 ? FD : 1], psiS[FD];
#pragma unroll
  for (int t = 0; t < FD; ++t) {
    psiX[t] = real(0);
    if (DIM == 3) psiY[t] = real(0);
    psiS[t] = bS;
  }

  // edge words: lane's word number u of the x edge belongs to tile row u / FW, of
  // the y edge to tile column u / FW; a row's plane at step s is s - row
  const bool rx = tx > 0, ry = DIM == 3 && ty > 0;                          // (uniform)
  const bool px = tx + 1 < a.tiles_x, py = DIM == 3 && ty + 1 < a.tiles_y;  // (uniform)
  const unsigned long long* in_x = a.edge_x + ((size_t)d * tiles + tile - 1) * NS * WY * FW;
  const unsigned long long* in_y = a.edge_y + ((size_t)d * tiles + tile - a.tiles_x) * NS * WX * FW;
  unsigned long long* out_x = a.edge_x + ((size_t)d * tiles + tile) * NS * WY * FW;
  unsigned long long* out_y = a.edge_y + ((size_t)d * tiles + tile) * NS * WX * FW;
  unsigned long long rX[NEX], rY[NEY ? NEY : 1];
#pragma unroll
  for (int k = 0; k < NEX; ++k) rX[k] = 0;
#pragma unroll
  for (int k = 0; k < (NEY ? NEY : 1); ++k) rY[k] = 0;
  // word u = lane + 32 k of an edge with E cells: its cell, valid, on the mesh
  auto edge_cell = [&](int k) { return (lane + 32 * k) / FW; };
  auto fetch = [&](const unsigned long long* in, int E, int step, int k, int limit) -> unsigned long long {
    const int e = edge_cell(k), r = step - e;  // (the edge's cells are skewed by their own position)
    if (e < E && e < limit && (unsigned)r < (unsigned)NS) return ld_relaxed_u64(in + (long)r * E * FW + lane + 32 * k);
    return 0;
  };
  const int rows_ok = DIM == 3 ? NY - ty * WY : 1, cols_ok = NX - tx * WX;  // tile rows / columns on the mesh

  const int nsteps = NS + WX - 1 + WY - 1;
  int slot = 0, fill = S::PF;
  unsigned on = active(0), on1 = active(1);  // the cells with a plane at this step and the next
  static_assert(S::PF == 2, "on, on1, on2");
  for (int s = 0; s < nsteps; ++s) {
    const int sc = s - skew;
    const bool act = col_ok && (unsigned)sc < (unsigned)NS;
    const unsigned on2 = active(s + 2);
    // ---- upwind tile's outflow into the edge slots
    bool failed = false;
    if (rx) {
#pragma unroll
      for (int k = 0; k < NEX; ++k) {
        const int u = lane + 32 * k, e = edge_cell(k), r = s - e;
        if (e < WY && e < rows_ok && (unsigned)r < (unsigned)NS) {
          const unsigned tag = want_epoch | (unsigned)r;
          unsigned v = (unsigned)rX[k];
          if ((unsigned)(rX[k] >> 32) != tag)
            failed |= !poll_word(in_x + (long)r * WY * FW + u, tag, &v, a.status, a.wait_limit_ns);
          *reinterpret_cast<unsigned*>(sm + S::o_ex + e * S::EB + (u - e * FW) * 4) = v;
        }
      }
    }
    if (DIM == 3 && ry) {
#pragma unroll
      for (int k = 0; k < NEY; ++k) {
        const int u = lane + 32 * k, e = edge_cell(k), r = s - e;
        if (e < WX && e < cols_ok && (unsigned)r < (unsigned)NS) {
          const unsigned tag = want_epoch | (unsigned)r;
          unsigned v = (unsigned)rY[k];
          if ((unsigned)(rY[k] >> 32) != tag)
            failed |= !poll_word(in_y + (long)r * WX * FW + u, tag, &v, a.status, a.wait_limit_ns);
          *reinterpret_cast<unsigned*>(sm + S::o_ey + e * S::EB + (u - e * FW) * 4) = v;
        }
      }
    }
    if ((rx || ry) && __any_sync(FULL, failed)) {  // status is set; drain own copies, leave
      cp_async_wait<0>();
      break;
    }
    // the next plane's words, one step ahead (tags are checked when used)
    if (rx) {
#pragma unroll
      for (int k = 0; k < NEX; ++k) rX[k] = fetch(in_x, WY, s + 1, k, rows_ok);
    }
    if (DIM == 3 && ry) {
#pragma unroll
      for (int k = 0; k < NEY; ++k) rY[k] = fetch(in_y, WX, s + 1, k, cols_ok);
    }
    cp_async_wait<S::PF - 1>();  // this step's sources have landed
    __syncwarp();
    // ---- upwind face values: the neighbour's outflow, or the edge slot's
    real upX[FD], upY[DIM == 3 ? FD : 1], ex[S::EB / SZ], ey[S::EB / SZ];
    load_edge<S::kDirect, FD>(ex, sm + S::o_ex + ly * S::EB);
    if (DIM == 3) load_edge<S::kDirect, FD>(ey, sm + S::o_ey + lx * S::EB);
#pragma unroll
    for (int t = 0; t < FD; ++t) {
      const real sx = A::shfl_up(psiX[t], 1);
      upX[t] = lx == 0 ? ex[t] : sx;
      if constexpr (DIM == 3) {
        const real sy = A::shfl_up(psiY[t], WX);
        upY[t] = ly == 0 ? ey[t] : sy;
      }
    }
    // ---- material of this plane (class 0 for idle lanes)
    const unsigned char* Ai = ainv;
    {
      const unsigned char* at = sm + S::o_cls + lane * 4;
      const unsigned cls = bytes ? at[((sc >> 2) & (S::CW - 1)) * 128 + (sc & 3)]
                                 : *reinterpret_cast<const unsigned*>(at + (sc & (S::CW - 1)) * 128);
      Ai += (size_t)(act ? cls : 0u) * ainv_class;
    }
    // the first columns of the inverse, on their way while b is formed
    constexpr int PJ = 8 / SZ, PL = 16 / SZ;  // columns per piece of a row pair, of the lone row
    constexpr int NCP = RW::pair_pieces(SZ);
    // pieces of each row pair in flight (Apply, us, with 0 / 1 / 2 / 3: 3-D Q1 64^3
    // GLC S12 3993 / 3697 / 3908 / 4157, where registers are short; 2-D Q1 32^2
    // 105 / 102 / 100 / -; FP32 3-D Q1 128^3 5382 / 5471 / 5552)
    constexpr int AHEAD = SZ == 4 ? 0 : N == 8 ? 1 : 2;
    uint4 ring[AHEAD ? AHEAD : 1][RP];
#pragma unroll
    for (int c = 0; c < AHEAD; ++c)
#pragma unroll
      for (int p = 0; p < RP; ++p) ring[c][p] = ldg_first(Ai + 16 * (p * NCP + c));
    // ---- right-hand side
    real b[N];
    {
      const unsigned char* src = sm + S::o_src + (slot * arrays * 32 + lane) * S::SRC;
      const unsigned char* isrc = src + 32 * S::SRC;
      int o0 = 0, o1 = 0;
      if (!kAligned) {
        const long cb = (long)(col + cell0 + (s - skew) * cstep) * S::CELLB;
        o0 = (int)((reinterpret_cast<size_t>(src0) + cb) & 15);
        if (FM >= 1) o1 = (int)((reinterpret_cast<size_t>(a.iso) + cb) & 15);
      }
      if constexpr (S::kDirect) {  // 16 bytes at a time: pairs at a stride of 48 bytes met two-way conflicts
        P v[N / 2];
        auto fetch_cell = [&](const unsigned char* from) {
#pragma unroll
          for (int c = 0; c < N / 4; ++c) {
            const uint4 u = *reinterpret_cast<const uint4*>(from + 16 * c);
            K::from16(u, v + 2 * c);
          }
          flip_pairs(v, flip);
        };
        typename K::Acc acc[N / 2];
        if (FM >= 1) {
          if (arrays == 2) fetch_cell(isrc);
#pragma unroll
          for (int m = 0; m < N / 2; ++m) acc[m] = K::from(arrays == 2 ? v[m] : K::make(real(0), real(0)));
        }
        fetch_cell(src);
#pragma unroll
        for (int m = 0; m < N / 2; ++m) {
          if (FM >= 1) {
            K::fma(acc[m], K::make(w0, w0), K::op(v[m]), z);
            v[m] = K::raw(acc[m]);
          }
          b[2 * m] = K::get(v[m], 0);
          b[2 * m + 1] = K::get(v[m], 1);
        }
      } else if constexpr (P1 == 2) {
#pragma unroll
        for (int m = 0; m < N / 2; ++m) {
          const int at = (phys(2 * m) - (swap ? 1 : 0)) * SZ;
          P v = K::swap_if(K::array_load(src + at), swap);
          if (FM >= 1) {
            typename K::Acc acc = K::from(arrays == 2 ? K::swap_if(K::array_load(isrc + at), swap)
                                                      : K::make(real(0), real(0)));
            K::fma(acc, K::make(w0, w0), K::op(v), z);
            v = K::raw(acc);
          }
          b[2 * m] = K::get(v, 0);
          b[2 * m + 1] = K::get(v, 1);
        }
      } else {
#pragma unroll
        for (int i = 0; i < N; ++i) {
          const int at = phys(i) * SZ;
          b[i] = *reinterpret_cast<const real*>(src + o0 + at);
          if (FM >= 1) {
            typename A::acc acc = A::from(arrays == 2 ? *reinterpret_cast<const real*>(isrc + o1 + at) : real(0));
            A::fma(acc, w0, b[i]);
            b[i] = A::raw(acc);
          }
        }
      }
    }
    // face products and terms.  2-D: row t of the x face with row t of the
    // sweep-axis face; dof 0 lies on both faces and takes its x term first
    if constexpr (DIM == 2) {
      const P* F = reinterpret_cast<const P*>(a.facep);  // [t][u] = (F_x, F_S)
      typename K::Op up[FD];
#pragma unroll
      for (int u = 0; u < FD; ++u) up[u] = K::op(K::make(upX[u], psiS[u]));
#pragma unroll
      for (int t = 0; t < FD; ++t) {
        typename K::Acc acc = K::prod(F[t * FD], up[0], z);
#pragma unroll
        for (int u = 1; u < FD; ++u) K::fma(acc, F[t * FD + u], up[u], z);
        const P f = K::raw(acc);
        if (t == 0) {
          typename A::acc s0 = A::from(b[0]);
          A::fma(s0, wX, K::get(f, 0));
          s0 = A::from(A::raw(s0));
          A::fma(s0, wS, K::get(f, 1));
          b[0] = A::raw(s0);
        } else {
          typename K::Acc sp = K::from(K::make(b[C::x_in(t)], b[C::s_in(t)]));
          K::fma(sp, K::make(wX, wS), K::op(f), z);
          const P v = K::raw(sp);
          b[C::x_in(t)] = K::get(v, 0);
          b[C::s_in(t)] = K::get(v, 1);
        }
      }
    } else {
      // rows 2m and 2m + 1 of each face: x dofs (0, 2), (4, 6), sweep-axis dofs
      // (0, 1), (2, 3), y dofs (0, 1), (4, 5); a dof takes its x, sweep-axis, y terms
      static_assert(DIM == 2 || P1 == 2, "3-D: Q1 cells");
      const P* F = reinterpret_cast<const P*>(a.facep);  // [x, S, y][m][u] = rows (2m, 2m + 1)
#pragma unroll
      for (int ax = 0; ax < 3; ++ax) {
        const real w = ax == 0 ? wX : (ax == 1 ? wS : wY);
        typename K::Op up[FD];
#pragma unroll
        for (int u = 0; u < FD; ++u) {
          const real v = ax == 0 ? upX[u] : (ax == 1 ? psiS[u] : upY[DIM == 3 ? u : 0]);
          up[u] = K::op(K::make(v, v));
        }
#pragma unroll
        for (int m = 0; m < FD / 2; ++m) {
          typename K::Acc acc = K::prod(F[(ax * (FD / 2) + m) * FD], up[0], z);
#pragma unroll
          for (int u = 1; u < FD; ++u) K::fma(acc, F[(ax * (FD / 2) + m) * FD + u], up[u], z);
          const int i0 = ax == 0 ? C::x_in(2 * m) : (ax == 1 ? C::s_in(2 * m) : C::y_in(2 * m));
          const int i1 = ax == 0 ? C::x_in(2 * m + 1) : (ax == 1 ? C::s_in(2 * m + 1) : C::y_in(2 * m + 1));
          typename K::Acc sp = K::from(K::make(b[i0], b[i1]));
          K::fma(sp, K::make(w, w), K::op(K::raw(acc)), z);
          const P v = K::raw(sp);
          b[i0] = K::get(v, 0);
          b[i1] = K::get(v, 1);
        }
      }
    }
    issue(fill, s + S::PF, on2);  // refills the slot consumed a step ago
    if (!bytes || (s & 3) == 0) class_word((bytes ? sc >> 2 : sc) + 2);  // (needed two or more steps later)
    cp_async_commit();
    slot = slot + 1 == S::RING ? 0 : slot + 1;
    fill = fill + 1 == S::RING ? 0 : fill + 1;
    // ---- x = A'^-1 b
    real x[N];
    {
      typename K::Op bp[N];
#pragma unroll
      for (int j = 0; j < N; ++j) bp[j] = K::op(K::make(b[j], b[j]));
      typename K::Acc acc[RP];
#pragma unroll
      for (int c = 0; c < NCP; ++c) {
#pragma unroll
        for (int p = 0; p < RP; ++p) {
          P row[PJ];
          if constexpr (AHEAD > 0) {
            K::from16(ring[c % (AHEAD ? AHEAD : 1)][p], row);
            if (c + AHEAD < NCP) ring[c % (AHEAD ? AHEAD : 1)][p] = ldg_first(Ai + 16 * (p * NCP + c + AHEAD));
          } else {
            K::from16(ldg_keep(reinterpret_cast<const uint4*>(Ai + 16 * (p * NCP + c))), row);
          }
#pragma unroll
          for (int j = 0; j < PJ; ++j) {
            const int cl = c * PJ + j;
            if (cl == 0) acc[p] = K::prod(row[0], bp[0], z);
            else if (cl < N) K::fma(acc[p], row[j], bp[cl < N ? cl : 0], z);
          }
        }
      }
#pragma unroll
      for (int p = 0; p < RP; ++p) {
        const P v = K::result(acc[p]);
        x[2 * p] = K::get(v, 0);
        x[2 * p + 1] = K::get(v, 1);
      }
      if constexpr (kOdd) {
        typename A::acc al = A::zero();
#pragma unroll
        for (int c = 0; c < RW::lone_pieces(SZ); ++c) {
          real l[PL];
          load_row<real, PL>(reinterpret_cast<const real*>(Ai + 16 * (RP * NCP + c)), l);
#pragma unroll
          for (int j = 0; j < PL; ++j) {
            const int cl = c * PL + j;
            if (cl == 0) al = A::prod(l[0], b[0]);
            else if (cl < N) A::fma(al, l[j], b[cl < N ? cl : 0]);
          }
        }
        x[N - 1] = A::get(al);
      }
    }
    if (act) {
#pragma unroll
      for (int t = 0; t < FD; ++t) {
        psiX[t] = x[C::x_out(t)];
        psiS[t] = x[C::s_out(t)];
        if (DIM == 3) psiY[DIM == 3 ? t : 0] = x[C::y_out(t)];
      }
    }
    // ---- the cells' values, in physical order: to memory, the tile's outflow to its
    // slot; or all into the shared slot
    if constexpr (S::kDirect) {
      if (px && lx == WX - 1)
        for (int t = 0; t < FD; ++t) *reinterpret_cast<real*>(sm + S::o_ox + ly * S::EB + t * SZ) = x[C::x_out(t)];
      if (DIM == 3 && py && ly == WY - 1)
        for (int t = 0; t < FD; ++t) *reinterpret_cast<real*>(sm + S::o_oy + lx * S::EB + t * SZ) = x[C::y_out(t)];
    } else {
      unsigned char* out = sm + lane * S::OUT;
      if constexpr (P1 == 2) {
#pragma unroll
        for (int m = 0; m < N / 2; ++m)
          K::array_put(out + (phys(2 * m) - (swap ? 1 : 0)) * SZ, K::swap_if(K::make(x[2 * m], x[2 * m + 1]), swap));
      } else {
#pragma unroll
        for (int i = 0; i < N; ++i) *reinterpret_cast<real*>(out + phys(i) * SZ) = x[i];
      }
    }
    __syncwarp();
    // ---- outflow of the tile's last cells first (the downwind tiles wait on it), then psi
    if (px) {
#pragma unroll
      for (int k = 0; k < NEX; ++k) {
        const int u = lane + 32 * k, e = edge_cell(k), r = s - (WX - 1) - e, g = e * WX + WX - 1;
        if (e < WY && ((on >> (g & 31)) & 1u)) {
          const int w = u - e * FW, i = phys(C::x_out(w / W)) * W + w % W;
          const unsigned v = *reinterpret_cast<const unsigned*>(sm + (S::kDirect ? S::o_ox + e * S::EB + w * 4 : g * S::OUT + i * 4));
          st_relaxed_u64(out_x + (long)r * WY * FW + u, ((unsigned long long)((a.epoch << 16) | (unsigned)r) << 32) | v);
        }
      }
    }
    if (DIM == 3 && py) {
#pragma unroll
      for (int k = 0; k < NEY; ++k) {
        const int u = lane + 32 * k, e = edge_cell(k), r = s - (WY - 1) - e, g = (WY - 1) * WX + e;
        if (e < WX && ((on >> (g & 31)) & 1u)) {
          const int w = u - e * FW, i = phys(C::y_out(w / W)) * W + w % W;
          const unsigned v = *reinterpret_cast<const unsigned*>(sm + (S::kDirect ? S::o_oy + e * S::EB + w * 4 : g * S::OUT + i * 4));
          st_relaxed_u64(out_y + (long)r * WX * FW + u, ((unsigned long long)((a.epoch << 16) | (unsigned)r) << 32) | v);
        }
      }
    }
    const int adv = s * cstep;
    if constexpr (S::kDirect) {
      P v[N / 2];
#pragma unroll
      for (int m = 0; m < N / 2; ++m) v[m] = K::make(x[2 * m], x[2 * m + 1]);
      flip_pairs(v, flip);
      if (act)
        store_cell(reinterpret_cast<unsigned char*>(a.psi + dirbase) + (long)(col + cell0 + (s - skew) * cstep) * S::CELLB, v);
    } else if constexpr (kAligned) {  // (the pieces are the source copies')
      unsigned char* pout = reinterpret_cast<unsigned char*>(a.psi + dirbase);
      auto piece = [&](int j) {
        const int u = lane + 32 * j, g = u / CH, p = u - g * CH;
        const uint4 v = *reinterpret_cast<const uint4*>(sm + g * S::OUT + 16 * p);
        __stcs(reinterpret_cast<uint4*>(pout + (long)(sc_cell[j] + adv) * S::CELLB + 16 * p), v);
      };
      if (on == FULL) {
#pragma unroll
        for (int j = 0; j < CH; ++j) piece(j);
      } else {
#pragma unroll
        for (int j = 0; j < CH; ++j)
          if ((on >> ((lane + 32 * j) / CH)) & 1u) piece(j);
      }
    } else {
      real* pout = a.psi + dirbase + (long)adv * N;
      const real* from = reinterpret_cast<const real*>(sm) + lane;
      if (on == FULL) {
#pragma unroll
        for (int j = 0; j < NP; ++j) store_stream(pout + po[j], from[32 * j]);
      } else {
#pragma unroll
        for (int j = 0; j < NP; ++j)
          if ((on >> ((lane + 32 * j) / N)) & 1u) store_stream(pout + po[j], from[32 * j]);
      }
    }
    on = on1;
    on1 = on2;
  }
}

// resident blocks per SM the registers are cut for
template <typename real, int DIM, int P1>
constexpr int lane_blocks() {
  constexpr int N = Cell<DIM, P1>::N;
  // (3-D Q1, Apply, us: FP32 128^3 with 3 / 4 / 5 / 6 blocks 6057 / 5382 / 5229 / 5913,
  // FP64 64^3 with 3 / 4 blocks 3697 / 4707)
  return sizeof(real) == 8 ? (N == 4 ? 4 : N == 8 ? 3 : 2) : (N == 4 ? 6 : N == 8 ? 5 : 4);
}
template <typename real, int DIM, int P1, int FM>
__global__ void __launch_bounds__(128, (lane_blocks<real, DIM, P1>())) sweep_lane_kernel(const __grid_constant__ SweepArgs<real> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr unsigned FULL = 0xffffffffu;
  for (;;) {
    int task = 0, stop = 0;
    if ((threadIdx.x & 31) == 0) {
      task = atomicAdd(a.ticket, 1);
      stop = *(volatile int*)a.status;
    }
    task = __shfl_sync(FULL, task, 0);
    stop = __shfl_sync(FULL, stop, 0);
    if (task >= a.n_tasks || stop) return;
    sweep_lane_task<real, DIM, P1, FM>(a, task, smem_raw);
  }
}

// Many problems in one persistent launch (see sweep_batch_kernel)
template <typename real, int DIM, int P1, int FM>
__global__ void __launch_bounds__(128, (lane_blocks<real, DIM, P1>()))
    sweep_lane_batch_kernel(const SweepArgs<real>* __restrict__ args, const int2* __restrict__ tmap, int n_total,
                            int* ticket, const int* status, const unsigned* epoch) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ SweepArgs<real> s_args[4];
  for (;;) {
    const int p = next_batch_task(args, tmap, n_total, ticket, status, epoch, s_args[threadIdx.x >> 5]);
    if (p < 0) return;
    sweep_lane_task<real, DIM, P1, FM>(s_args[threadIdx.x >> 5], p, smem_raw);
    __syncwarp();  // the slot is rewritten by the next task
  }
}

template <typename real, int DIM, int P1, int FM>
cudaError_t launch_lane_fm(const SweepArgs<real>& a, int grid, int block, cudaStream_t s) {
  using S = LaneSlot<real, DIM, P1>;
  const int arrays = FM >= 1 && a.iso ? 2 : 1;
  const size_t warps = block / 32, smem = warps * S::bytes(arrays);
  static SweepLaunch st;
  const cudaError_t e = st.prepare((const void*)sweep_lane_kernel<real, DIM, P1, FM>, arrays, grid, block, smem,
                                   warps * S::bytes(FM >= 1 ? 2 : 1), 0, kGroupKeepKb);
  if (e != cudaSuccess) return e;
  sweep_lane_kernel<real, DIM, P1, FM><<<grid, block, smem, s>>>(a);
  return cudaGetLastError();
}
template <typename real, int DIM, int P1, int FM>
cudaError_t launch_lane_batch_fm(const BatchLaunch<real>& b, cudaStream_t s) {
  using S = LaneSlot<real, DIM, P1>;
  const int arrays = FM >= 1 && b.sources ? 2 : 1;
  const size_t warps = b.block / 32, smem = warps * S::bytes(arrays);
  static SweepLaunch st;
  const cudaError_t e = st.prepare((const void*)sweep_lane_batch_kernel<real, DIM, P1, FM>, arrays, b.grid, b.block, smem,
                                   warps * S::bytes(FM >= 1 ? 2 : 1), 4 * sizeof(SweepArgs<real>), kGroupKeepKb);
  if (e != cudaSuccess) return e;
  sweep_lane_batch_kernel<real, DIM, P1, FM>
      <<<b.grid, b.block, smem, s>>>(b.args, b.tmap, b.n_total, b.ticket, b.status, b.epoch);
  return cudaGetLastError();
}

template <typename real, int DIM>
cudaError_t launch_lane_dim(int p1, int fm, const SweepArgs<real>& a, int grid, int block, cudaStream_t s) {
  if (fm != 0 && fm != 1) return cudaErrorInvalidValue;
  if (p1 == 2)
    return fm ? launch_lane_fm<real, DIM, 2, 1>(a, grid, block, s) : launch_lane_fm<real, DIM, 2, 0>(a, grid, block, s);
  if constexpr (DIM == 2)
    if (p1 == 3)
      return fm ? launch_lane_fm<real, 2, 3, 1>(a, grid, block, s) : launch_lane_fm<real, 2, 3, 0>(a, grid, block, s);
  return cudaErrorInvalidValue;
}
template <typename real, int DIM>
cudaError_t launch_lane_batch_dim(int p1, int fm, const BatchLaunch<real>& b, cudaStream_t s) {
  if (fm != 0 && fm != 1) return cudaErrorInvalidValue;
  if (p1 == 2) return fm ? launch_lane_batch_fm<real, DIM, 2, 1>(b, s) : launch_lane_batch_fm<real, DIM, 2, 0>(b, s);
  if constexpr (DIM == 2)
    if (p1 == 3) return fm ? launch_lane_batch_fm<real, 2, 3, 1>(b, s) : launch_lane_batch_fm<real, 2, 3, 0>(b, s);
  return cudaErrorInvalidValue;
}

}  // namespace ouranos
