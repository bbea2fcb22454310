// lbm_quad.cuh — the 16-bit AA step over quad rows (kRowsQuad).
//
// Quad rows store the 8-byte word w of a row (0 <= w < D, D = px/4) as the
// nodes w, w + 2D, w + D, w + 3D in its four 16-bit slots: the low 32-bit
// half is the paired word (w, w + H) and the high half the paired word
// (w + D, w + D + H), H = px/2.  One thread takes one word, four nodes:
// both AA step kinds then touch every population as one aligned 8-byte
// word per thread (a warp moves 256 contiguous bytes per access), because
// a node one step away in x is one word away for all four nodes.  The node
// arithmetic runs twice, once per half, on F2 lanes (packed FP32) — the
// arithmetic of the paired pull step, which the 16-bit units compile
// without multiply-add contraction, so a node gets the same bits as from
// the per-node AA step over plain rows.
//
// Local step (natural -> swapped): word w of plane q in, word w of plane
// opp q out, all at the node.  Channels: the pending natural slots of the
// inlet (x = 0: slot 0 of word 0) and the outlet (x = nx - 1: slot 3 of word
// D - 1) take their open-face rules first, as in the per-node step.
//
// Neighbour step (swapped -> natural): population q of the four nodes is
// read from word w - c_x of the donor row in plane opp q and written to word
// w + c_x of the destination row in plane q.  The words that differ:
//   - seams: for word 0 with c_x = +1 the nodes x - 1 lie in word D - 1 one
//     slot down (kD - 1 = (D - 1) + (k - 1) D), and node 0's donor is outside
//     the box: the node's own slot (0, q), with the node's wall rule; for
//     word D - 1 with c_x = -1 likewise in word 0 one slot up, node nx - 1's
//     donor outside.  The stores mirror this: word 0 with c_x = -1 writes
//     three slots of word D - 1 (one 32-bit and one 16-bit store) and node
//     0's value into its own slot (0, opp q); word D - 1 with c_x = +1 writes
//     three slots of word 0 and node nx - 1's own slot.  Only these two
//     threads of a row branch, and only for the five populations with that
//     c_x.  Slot ownership makes the split stores race-free: in a neighbour
//     step every slot is read and written by one node only (x - c_p for slot
//     (x, p), or the node itself when that lies outside), so the slots of
//     word D - 1 that thread 0 writes are disjoint from the one that thread
//     D - 1 writes, and every whole-word store covers slots of its own four
//     nodes only (px == nx: no padding nodes).
//   - rows on a y or z face: a population whose donor row is outside reads
//     the node's own word of plane q and takes each node's wall rule; one
//     whose destination row is outside writes the node's own word of plane
//     opp q with each node's wall value (aa_wall).
// No word is read outside its plane's rows: a seam word is addressed in its
// own row, never one word past the row.
#pragma once
#include "lbm_kernels.cuh"

namespace lbm {

// the word AA step applies to the domain's geometry (quad rows, no STRUCT
// nodes, px == nx: no padding nodes)
__host__ __device__ __forceinline__ bool aa_words_apply(const Geometry& g) {
  return g.rows == kRowsQuad && !has_struct(g) && g.px == g.nx && g.nx >= 16;
}

__device__ __forceinline__ uint2 ld_w8(const void* p) {
  return *reinterpret_cast<const uint2*>(p);
}
__device__ __forceinline__ void st_w8(void* p, uint2 v) { *reinterpret_cast<uint2*>(p) = v; }
__device__ __forceinline__ void st_w4(void* p, uint32_t v) {
  *reinterpret_cast<uint32_t*>(p) = v;
}
__device__ __forceinline__ void st_w2(void* p, uint32_t v) {
  *reinterpret_cast<unsigned short*>(p) = (unsigned short)v;
}

// Resident threads per SM the register budget is sized for (two F2 halves per
// thread, 128 registers).
#ifndef LBM_QUAD_THREADS_PER_SM
#define LBM_QUAD_THREADS_PER_SM 512
#endif

// One AA step (NB = 0 local, 1 neighbour) of the four nodes of word w of row
// (y, z).  Slot tables as for the per-node AA step (aa_args with a.off[q] =
// 4 c_x + px (c_z + nz c_y)): local srcd[q] = plane q, dstq[q] = plane opp q;
// neighbour srcd[q] = plane opp q - off_q, dstq[q] = plane q + off_q; srcq[q] =
// plane q.  entry (local steps): kAAPending or kAAComplete (the first step
// after the initial state is the per-node step's).
// FACE (neighbour step): the row may lie on a y or z face, so that some
// populations' donor or destination rows are outside the box; the rows off
// the faces are stepped by CTAs without that code (FACE = false).
// MACRO: only rho and u of arF in the layout that step would read, for
// a.den_out and a.ux_out.
template <class S, int COLL, bool LES, bool SR, int NB, bool FACE, bool MACRO = false>
__device__ __forceinline__ void aa_word(const StepArgs<S>& a, int w, int y, int z, int entry) {
  static_assert(kDev<S>, "quad rows are a 16-bit layout");
  static_assert(NB || !FACE, "face rows matter to the neighbour step only");
  const int D = a.g.px >> 2, H = a.g.px >> 1;
  const int e = 4 * w + a.g.px * (z + a.g.nz * y);  // slot 0 of the word
  const bool seam_lo = w == 0, seam_hi = w == D - 1;
  // donor / destination row of population q inside the box (rows off a
  // face: always)
  auto row_in = [&](int dy, int dz) {
    if constexpr (!FACE) return true;
    return (unsigned)(y + dy) < (unsigned)a.g.ny && (unsigned)(z + dz) < (unsigned)a.g.nz;
  };
  uint2 v[Q];
  if constexpr (!NB) {
    static_for<0, Q>([&](auto qc) {
      constexpr int q = decltype(qc)::value;
      v[q] = ld_w8(a.srcd[q] + e);
    });
  } else {
    static_for<0, Q>([&](auto qc) {
      constexpr int q = decltype(qc)::value;
      // the donor word w - c_x, or across the seam the word at the other end
      // of the same donor row (px elements away); a donor row outside: the
      // own slots (x, q), which hold f*_{opp q}
      int adj = 0;
      if constexpr (cx(q) == 1) adj = seam_lo ? a.g.px : 0;
      if constexpr (cx(q) == -1) adj = seam_hi ? -a.g.px : 0;
      v[q] = ld_w8(row_in(-cy(q), -cz(q)) ? a.srcd[q] + (e + adj) : a.srcq[q] + e);
    });
    // seam words: the own word of the five populations is fetched for all of
    // them before the first is used (one memory latency; fetched one after
    // the other they made a 32^3 neighbour step 3.5 times its local step)
    if (seam_lo) {
      uint2 own[Q];
      static_for<0, Q>([&](auto qc) {
        constexpr int q = decltype(qc)::value;
        if constexpr (cx(q) == 1) own[q] = ld_w8(a.srcq[q] + e);
      });
      static_for<0, Q>([&](auto qc) {
        constexpr int q = decltype(qc)::value;
        if constexpr (cx(q) == 1) {
          // quarters (own k0, X k0, X k1, X k2) in slot order k0 k2 | k1 k3
          const uint2 X = v[q];
          v[q].x = __byte_perm(own[q].x, X.y, 0x5410);
          v[q].y = X.x;
          if (!row_in(-cy(q), -cz(q))) v[q] = own[q];
        }
      });
    }
    if (seam_hi) {
      uint2 own[Q];
      static_for<0, Q>([&](auto qc) {
        constexpr int q = decltype(qc)::value;
        if constexpr (cx(q) == -1) own[q] = ld_w8(a.srcq[q] + e);
      });
      static_for<0, Q>([&](auto qc) {
        constexpr int q = decltype(qc)::value;
        if constexpr (cx(q) == -1) {
          // quarters (X k1, X k2, X k3, own k3)
          const uint2 X = v[q];
          v[q].x = X.y;
          v[q].y = __byte_perm(X.x, own[q].y, 0x7632);
          if (!row_in(-cy(q), -cz(q))) v[q] = own[q];
        }
      });
    }
  }
  const uint32_t kstep = SR ? a.kctr[a.kpar] : 0u;
  // store of population q's word of results (slot order)
  auto store = [&](auto qc, uint2 r) {
    constexpr int q = decltype(qc)::value;
    if constexpr (!NB) {
      st_w8(a.dstq[q] + e, r);
    } else {
      if (!row_in(cy(q), cz(q))) {
        st_w8(a.dst + (opp(q) * a.qs + e), r);  // own slots (x, opp q)
      } else if (cx(q) == -1 && seam_lo) {
        // the word across the seam is the last one of the destination row:
        // its slots k0 k2 k1 <- results k1 k3 k2; quarter 0 (x = 0) to its
        // own slot
        S* wd = a.dstq[q] + (e + a.g.px);
        st_w4(wd, r.y);
        st_w2(wd + 2, r.x >> 16);
        st_w2(a.dst + (opp(q) * a.qs + e), r.x & 0xffffu);
      } else if (cx(q) == 1 && seam_hi) {
        // the word across the seam is the first one of the destination row:
        // its slots k2 k1 k3 <- results k0 k1 k2; quarter 3 (x = nx - 1) to
        // its own slot
        S* wd = a.dstq[q] + (e - a.g.px);
        st_w4(wd + 2, r.x);
        st_w2(wd + 1, r.y & 0xffffu);
        st_w2(a.dst + (opp(q) * a.qs + e + 3), r.y >> 16);
      } else {
        st_w8(a.dstq[q] + e, r);
      }
    }
  };
  // channels: inlet and outlet rules of node 0 (lo lane of half 0 of word 0,
  // c_x = +1 populations) and node nx - 1 (hi lane of half 1 of the last word,
  // c_x = -1 populations), in rows off the faces: f holds the node's own
  // f*_{opp q} there.  One lane of a row evaluates them; a kernel of its own
  // after each step, which left the values for the next one, cost a launch
  // and 10 scattered reads a row: 32^3 10.3 us a step against 4.8 here,
  // 256x72x64 26.8 against 20.9, 512x128x128 148 against 138.
  // What the rules read is fetched with the populations.
  const int yz = y * a.g.nz + z;
  const bool open_rows = !FACE && a.g.casetype == CHANNEL &&
                         (NB || (entry == kAAPending && y > 0 && y < a.g.ny - 1 && z > 0 &&
                                 z < a.g.nz - 1));
  [[maybe_unused]] float in_rho = 0.0f, in_u = 0.0f;
  [[maybe_unused]] float out_u[3] = {0.0f, 0.0f, 0.0f};
  if (open_rows) {
    if (seam_lo) {
      in_rho = a.prho_in[yz];
      in_u = mul_rn(-1.0f, a.inlet_u[yz]);  // c_d . u_in, c_d,x = -1
    }
    if (seam_hi) outlet_velocity<S>(a, yz, out_u);
  }
  auto open_face_rules = [&](F2 (&f)[Q], int hb) {
    if (hb == 0 && seam_lo) {
      static_for<0, Q>([&](auto qc) {
        constexpr int q = decltype(qc)::value;
        if constexpr (cx(q) == 1) f[q].v.x = inlet_value<S, q>(f[q].v.x, in_rho, in_u);
      });
    }
    if (hb == 1 && seam_hi) {
      static_for<0, Q>([&](auto qc) {
        constexpr int q = decltype(qc)::value;
        if constexpr (cx(q) == -1) f[q].v.y = outlet_value<S, q>(a, f[q].v.y, out_u);
      });
    }
  };
  // the cavity's lid, the only nodes of a face row whose rule changes the
  // value: y = ny - 1 off its edges
  [[maybe_unused]] const bool lid_row =
      FACE && a.g.casetype == CAVITY && y == a.g.ny - 1 && z > 0 && z < a.g.nz - 1;
  // the halves, each a compile-time pass: half hb holds the nodes
  // (w + hb D, w + hb D + H); the first leaves its packed results in its half
  // of v[q], the second stores each population's word as soon as its result
  // is known
  auto pass = [&](auto hbc) {
    constexpr int hb = decltype(hbc)::value;
    const int xlo = w + hb * D, xhi = xlo + H;
    [[maybe_unused]] const bool lid_lo = lid_row && !(hb == 0 && seam_lo);
    [[maybe_unused]] const bool lid_hi = lid_row && !(hb == 1 && seam_hi);
    F2 f[Q];
    static_for<0, Q>([&](auto qc) {
      constexpr int q = decltype(qc)::value;
      f[q] = unpack_pair<S>(hb ? v[q].y : v[q].x, a.inv_scale);
    });
    if constexpr (FACE) {
      if (lid_row) {
        static_for<0, Q>([&](auto qc) {
          constexpr int q = decltype(qc)::value;
          if constexpr (cy(q) == -1) {
            if (lid_lo) f[q].v.x = aa_wall<S>(a, NODE_MOVINGWALL, f[q].v.x, opp(q));
            if (lid_hi) f[q].v.y = aa_wall<S>(a, NODE_MOVINGWALL, f[q].v.y, opp(q));
          }
        });
      }
    } else {
      // channels: rows off the faces (neighbour step), the pending natural
      // slots of the inlet and outlet nodes (local step)
      if (open_rows) open_face_rules(f, hb);
    }
    PairState<F2> ps;
    make_pairs<F2, true>(f, ps);
    F2 ux, uy, uz;
    const F2 inv_rho = velocity<F2>(ps, ux, uy, uz);
    // (channels: the nodes 1, nx - 1 and nx - 2 leave their state for the rules)
    if (a.den_out || a.ux_out || (a.g.casetype == CHANNEL && (w == 1 || w >= D - 2))) {
      write_macro<S>(a, xlo, y, z, ps.rho_full.v.x, ux.v.x, uy.v.x, uz.v.x);
      write_macro<S>(a, xhi, y, z, ps.rho_full.v.y, ux.v.y, uy.v.y, uz.v.y);
    }
    if constexpr (MACRO) return;
    [[maybe_unused]] uint32_t h = 0u;
    if constexpr (SR) h = sr_hash((uint32_t)(xlo + H * (z + a.g.nz * y)), kstep, a.sr_seed);
    collide_node<S, COLL, LES, true, F2>(f, ps, ux, uy, uz, inv_rho, a, [&](auto qc, F2 r) {
      constexpr int q = decltype(qc)::value;
      if constexpr (FACE && cy(q) == 1) {
        // destination row outside: the wall value into the node's own slot
        if (lid_lo) r.v.x = aa_wall<S>(a, NODE_MOVINGWALL, r.v.x, q);
        if (lid_hi) r.v.y = aa_wall<S>(a, NODE_MOVINGWALL, r.v.y, q);
      }
      uint32_t p;
      if constexpr (SR)
        p = pack_pair_sr<S>(r, a.scale, sr_bits<q>(h));
      else
        p = pack_pair<S>(r, a.scale);
      if constexpr (hb == 0)
        v[q].x = p;
      else
        store(qc, make_uint2(v[q].x, p));
    });
  };
  pass(std::integral_constant<int, 0>{});
  pass(std::integral_constant<int, 1>{});
}

// number of rows on a y or z face: 2 nz at y = 0 and y = ny - 1, then
// 2 (ny - 2) at z = 0 and z = nz - 1
__host__ __device__ __forceinline__ int aa_face_rows(const Geometry& g) {
  return 2 * g.nz + 2 * (g.ny - 2);
}

// Neighbour step: CTA rows of the rows off the faces (blockIdx.y < ny - 2:
// plane 1 + blockIdx.y, its nz - 2 inner rows one behind the other), then the
// face rows, also one behind the other, in trailing CTAs (a CTA-uniform
// branch into the code with the face rules, so the hot code of the inner rows
// stays short and the face rows fill the grid's tail).
inline dim3 aa_neighbor_grid(const Geometry& g) {
  const long long D = g.px / 4, inner = D * (g.nz - 2), face = D * aa_face_rows(g);
  const long long fc = (face + 127) / 128, room = 65535 - (g.ny - 2);  // CTA rows left
  long long gx = (inner + 127) / 128;
  if (gx * room < fc) gx = (fc + room - 1) / room;
  return dim3((unsigned)gx, (unsigned)(g.ny - 2 + (fc + gx - 1) / gx), 1);
}

// Local step: grid = flat_grid, every row.  Neighbour step: grid =
// aa_neighbor_grid.  One word per thread, CTAs of 128 threads over words of
// consecutive rows (flat_item).  MACRO: rho and u instead of the step.
template <class S, int COLL, bool LES, bool SR, int NB, bool MACRO = false>
__global__ void __launch_bounds__(128, LBM_QUAD_THREADS_PER_SM / 128)
    k_aa_words(const __grid_constant__ StepArgs<S> a, int entry) {
  chain_wait();
  if constexpr (!MACRO) bump_step_counter<SR>(a);
  if constexpr (!NB) {
    const FlatItem i = flat_item(a);
    if (i.in) aa_word<S, COLL, LES, SR, 0, false, MACRO>(a, i.x, i.y, i.z, entry);
  } else if ((int)blockIdx.y < a.g.ny - 2) {
    // backwards with a.rev, as flat_item
    const unsigned t = (a.rev ? gridDim.x - 1 - blockIdx.x : blockIdx.x) * 128u + threadIdx.x;
    const int r = (int)fastdiv(t, a.mrow);
    if (r < a.g.nz - 2)
      aa_word<S, COLL, LES, SR, 1, false, MACRO>(
          a, (int)t - r * a.ri, a.rev ? a.g.ny - 2 - (int)blockIdx.y : 1 + (int)blockIdx.y, r + 1,
          entry);
  } else {
    const unsigned c = (blockIdx.y - (unsigned)(a.g.ny - 2)) * gridDim.x + blockIdx.x;
    const unsigned t = c * 128u + threadIdx.x;
    const int r = (int)fastdiv(t, a.mrow);
    if (r >= aa_face_rows(a.g)) return;
    int y, z;
    if (r < 2 * a.g.nz) {
      y = r < a.g.nz ? 0 : a.g.ny - 1;
      z = r < a.g.nz ? r : r - a.g.nz;
    } else {
      const int r2 = r - 2 * a.g.nz;
      z = r2 < a.g.ny - 2 ? 0 : a.g.nz - 1;
      y = 1 + (r2 < a.g.ny - 2 ? r2 : r2 - (a.g.ny - 2));
    }
    aa_word<S, COLL, LES, SR, 1, true, MACRO>(a, (int)t - r * a.ri, y, z, entry);
  }
}

}  // namespace lbm
