// Sweep-front kernel for complex64 and bf16-split factors in symmetric tiles:
// every cell solve of one front of the L-sweep preconditioner in one launch.
//
// The solve is the twisted block LU of kernels_sweep.cu (two half chains that
// meet at the middle line).  The cell matrix is complex symmetric up to a
// diagonal scaling: the x-couplings are scalars, and the y-couplings lo_j, hi_j
// are the same for every line, so E^-1 D_k E is symmetric for every line's
// diagonal block with e_j / e_{j-1} = (lo_j / hi_{j-1})^(1/2), and so are the
// inverted Schur complements E^-1 S_k^-1 E.  The factor holds only their lower
// halves, in 16 x 16 tiles (tile (I, J), I >= J; the diagonal tiles whole), and
// the solve runs on E^-1 x: right-hand sides are scaled by 1 / e_j where they
// are formed and solutions by e_j where they are stored.  A tile below the
// diagonal serves the product twice, as itself (rows of I with the input of J)
// and transposed (rows of J with the input of I), so a solve streams half the
// bytes of the whole blocks.
//
// Tile (I, J) of a line sits in class (I + J) mod 4, the classes one after the
// other, each by column (SymTable).  complex64: element (i, j) of a tile at
// 16 j + (i ^ f(j)), f(j) = 4 (j mod 4) + j / 4, so that 16 rows of a column and
// 16 columns of a row lie in distinct shared-memory banks.  split: four planes
// (real hi, imaginary hi, real lo, imaginary lo) of four 8 x 8 bf16 matrices, the
// form ldmatrix reads, as it is or transposed, straight into mma fragments.
//
// Work split.  An item (a cell and up to 16 right-hand-side slots) runs on a
// cluster of 2 CL CTAs, CL per half chain.  CTA c of a half streams 4 / CL of
// the classes: every row of tiles finds about 1 / CL of its tiles there, so
// the CTAs and, within a CTA, the consumer warps (one per 16 rows) are loaded
// alike.  A warp forms its rows' partial sums in registers:
//   complex64: lane = (row, even or odd columns of each tile), or up to 4 slots
//              (two rows, every fourth column), FMAs, the parts added by shuffles;
//   split:     mma.sync m16n8k16, the four products of hi and lo words against
//              the input's hi and lo words, FP32 accumulation (the fourth, lo x
//              lo, halves the preconditioner's error: 9e-5 against 2e-4 at 163-
//              point cells).  Against whole blocks and three products the split's
//              own error is 0.72-0.87x in a cell solve and up to 1.23x in an apply,
//              since the two entries that a value serves share its rounding and
//              their errors add in what travels to and fro.  An apply's whole
//              error against complex128 is 1.04x at 33 points per line, 1.18x at 54
//              and 73, 1.06x at 129 and 1.00x from 163 on, where the FP32 inverse
//              dominates (means over 16 media, +-0.01).
// The partial sums go to every other CTA of the half (st.async into its shared
// memory, completing the transaction count of its per-line mbarrier); each CTA
// finishes every row, all in the same order, in the registers of the lanes
// that formed its own sums.  So a line costs one exchange, one CTA barrier and
// no pass through shared memory but its input vector (two buffers).  One warp
// streams the chunks (one to four classes) through a ring with cp.async.bulk;
// two lanes issue them, since a copy keeps its issuing thread busy for about 470
// cycles whatever its size (measured: 16 KB copies 35 bytes per cycle from one
// lane and 61 from two, 32 KB copies 122 from two).
//
// What bounds a line (163 to 171 points, 4 slots, one CTA per half, measured by
// leaving parts out): split 6.6k cycles, of which 3.6k the products (shared-
// memory reads 2.9k, mma 2.4k) and the rest instructions of one warp after
// another, ~5 cycles each; complex64 10k, of which 6.6k the products (FMA issue
// 5k; 9.7k with two rows per lane).  Whole blocks took 10.5k and 13.4k.  So the line's code is kept short:
// addresses precomputed, no branch per tile (predicated loads), nothing built
// per line that the item can build once.  Two CTAs per SM (72 registers) and
// sharing an input block among three row tiles were slower.
//
// A lane keeps the right-hand side of the next line (forward) or the stored
// y_k (backward) of its own elements in registers, loaded a line ahead; y_k and
// x_k go to a per-item scratch, from which the outputs are written once per
// item at the end, many points' loads in flight at once.
//
// Registers: 128 per thread (thirteen warps at most; all slot counts in one kernel),
// with 100-160 bytes of spill stores in complex64 and 212-488 in the split.
//
// Every wait is bounded, as in kernels_sweep.cu.
#pragma once
#include "common.cuh"
#include "internal.h"
#include "sweep_common.cuh"

namespace lsw {

namespace {

constexpr int kHdr = 256;             // barriers and the abort flag
constexpr int kRingMax = 8;           // ring stages
constexpr int kTileB = 2048;          // bytes of a tile: 256 values of 8 bytes
constexpr int kSymWarps = 1 + kSymTilesMax;   // producer + one consumer warp per 16 rows
constexpr int SK_NONE = 99;           // padding slot

// complex64 line input: values per point, a 16-byte pad at 16 slots so that the
// two columns a warp reads at once lie in distinct banks
__host__ __device__ constexpr int sym_xs(int R) { return R == 16 ? 18 : R; }
// complex64: rows per lane of a tile.  A lane with two rows reads the input for
// half as many columns, and a 16-byte read costs ~1.5 cycles of the SM's shared
// memory whether its addresses are two or eight (measured): 8 x 8 cells of
// 128^2, an apply with 2 slots per item 8.8 -> 8.0 ms, with 4 11.7 -> 11.3; with
// 8 slots (twice the sums: fewer reads in flight) 4 x 4 cells 13.0 -> 14.1, so
// there a lane keeps one row.
__host__ __device__ constexpr int sym_rows(int R) { return R <= 4 ? 2 : 1; }

// elements of a lane: (row, slot) pairs it finishes
template <int R, bool SPLIT> struct Lane {
  static constexpr int NT = (2 * R + 7) / 8;   // split: mma n-tiles (Re, Im interleaved per slot)
  static constexpr int NE = SPLIT ? 2 * NT : (R > 1 ? R / 2 : 1);
};
// split line input: bytes of a row (term, part, slot), 16 mod 32 so that the eight
// rows of a matrix lie in distinct banks; always the 192 points of 12 blocks, so
// that a block past the cell reads zeros
constexpr unsigned kSplitRow = 2 * 16 * kSymTilesMax + 16;
// bytes of a line-input buffer for n16 points
template <int R, bool SPLIT> __host__ __device__ constexpr int sym_input_bytes(int n16) {
  return SPLIT ? 4 * 4 * Lane<R, SPLIT>::NT * (int)kSplitRow : n16 * sym_xs(R) * 8;
}


__device__ __forceinline__ float2 lds_c(unsigned a) {
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a));
  return v;
}
// four 8 x 8 matrices of 16-bit values, lane l giving row l % 8 of matrix l / 8
__device__ __forceinline__ void ldsm4(unsigned (&r)[4], unsigned addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
__device__ __forceinline__ void stsm4_t(unsigned addr, const unsigned (&r)[4]) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(r[0]), "r"(r[1]),
               "r"(r[2]), "r"(r[3])
               : "memory");
}
// the four planes of a tile (512 bytes apart), transposed where tn; zeros where !on
__device__ __forceinline__ void ldsm4x4(unsigned (&e)[4][4], unsigned addr, unsigned on, unsigned tn) {
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.eq.u32 p, %5, 1;\n\tsetp.eq.u32 q, %5, 3;\n\t"
        "mov.u32 %0, 0;\n\tmov.u32 %1, 0;\n\tmov.u32 %2, 0;\n\tmov.u32 %3, 0;\n\t"
        "@p ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];\n\t"
        "@q ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];\n\t}"
        : "=&r"(e[p][0]), "=&r"(e[p][1]), "=&r"(e[p][2]), "=&r"(e[p][3])
        : "r"(addr + p * 512), "r"(on | (tn << 1)));
  }
}
__device__ __forceinline__ void mbar_arrive_at(unsigned bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void st_remote(unsigned addr, float2 v, unsigned bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(addr),
               "f"(v.x), "f"(v.y), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void st_remote2(unsigned addr, float2 v0, float2 v1, unsigned bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(addr),
               "f"(v0.x), "f"(v0.y), "f"(v1.x), "f"(v1.y), "r"(bar)
               : "memory");
}

// a slot's place in its group's sum, and the group's owned box and output
struct OutSlot {
  long long off;
  int k0, k1, j0, j1;
  int first, last;
};
__device__ __forceinline__ void red_add2(float2* p, float2 v) {
  asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(p), "f"(v.x), "f"(v.y) : "memory");
}

template <int R, int CL, bool SPLIT>
__device__ __forceinline__ void sym_body(const FrontArgs& a, const DevItem& it, const DevCell& cl, unsigned char* smem) {
  using C = float2;
  constexpr int NT = Lane<R, SPLIT>::NT, NE = Lane<R, SPLIT>::NE;
  constexpr int RP = 4 * NT;                   // split: slots of the line input, padded
  constexpr int RH = R > 1 ? R / 2 : 1;
  constexpr bool V4 = !SPLIT && RH % 2 == 0;   // a lane's slots as 16-byte pairs
  constexpr int CLT = 2 * CL, NQ = 4 / CL;     // CTAs per item, classes per CTA
  constexpr int XS = sym_xs(R);                // complex64: values per point of the line input
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nx = cl.nx, ny = cl.ny;
  const int nb = (ny + 15) >> 4, n16 = nb << 4;
  const int NS = a.stages, cpc = a.ksw;        // ring stages, classes per chunk
  const unsigned crk = cluster_rank();
  if (cluster_size() != (unsigned)CLT || crk != blockIdx.x % (unsigned)CLT) {
    // the launch did not form the clusters this kernel was configured for
    // (uniform over the CTA: every thread leaves before any barrier)
    if (tid == 0) atomicOr(a.err, 4);
    return;
  }
  const int half = (int)crk / CL;        // 0: top chain, 1: bottom chain
  const int me = (int)crk % CL;          // rank within the half
  const unsigned rbase = (unsigned)(half * CL);
  const int mid = (nx - 1) / 2;
  const int nf = half == 0 ? mid : nx - 1 - mid;      // forward lines of my half (>= 2: nx >= 5)
  // line li of my half: forward li < nf, the middle line li == nf, backward after
  auto line_k = [&](int li) {
    const int i = li < nf ? li : 2 * nf - li;
    if (li == nf) return mid;
    return half == 0 ? i : nx - 1 - i;
  };
  const int nline = 2 * nf + 1;
  const int klo = half == 0 ? 0 : mid + 1, khi = half == 0 ? mid : nx - 1;   // lines whose outputs I write
  const int NCW = nb, NCT = NCW * 32;    // consumer warps, threads
  const int nslot = it.slot_count;
  const int q_first = me * NQ;
  const SymTable& symt = *a.symt;
  // tile rows whose x_k and outputs I write
  const int w_lo = (me * nb + CL - 1) / CL, w_hi = ((me + 1) * nb + CL - 1) / CL;

  // ---- shared layout (identical in every CTA of the cluster) ----
  uint64_t* full = reinterpret_cast<uint64_t*>(smem);
  uint64_t* empty = full + kRingMax;
  uint64_t* pready = empty + kRingMax;   // [2]: every other CTA's partial sums have landed (CL > 1)
  uint64_t* exitb = pready + 2;          // cluster-wide "done with remote shared memory"
  uint64_t* xch = exitb + 1;             // the other half's last forward vector has landed in P
  uint64_t* fwdb = xch + 1;              // every CTA of the half has stored its y_k (CL > 1)
  volatile int* abort_flag = reinterpret_cast<volatile int*>(fwdb + 1);
  static_assert((2 * kRingMax + 5) * 8 + 4 <= kHdr, "barrier header");
  // the ring starts at a multiple of the tile size (as an address and as a shared-memory offset from a base that is
  // the same in every CTA): the accesses within a tile are formed by XOR
  const unsigned ring_off = ((saddr(smem) + kHdr + kTileB - 1) & ~(unsigned)(kTileB - 1)) - saddr(smem);
  const unsigned stage_bytes = (unsigned)a.chunk;
  unsigned off = ring_off + (unsigned)NS * stage_bytes;
  const unsigned x_off = off;            // the line input, two buffers
  const unsigned x_bytes = (unsigned)sym_input_bytes<R, SPLIT>(n16);
  off += 2 * x_bytes;
  const unsigned q_off = off;            // [2][CL - 1][n16][R] partial sums of the other CTAs, plane d - 1: of CTA me ^ d
  const unsigned q_plane = (unsigned)(n16 * R * 8);
  off += 2 * (CL - 1) * q_plane;
  const unsigned p_off = off;            // [n16][R] the other half's y_{m-1} / z_{m+1}
  off += q_plane;
  C* wsh = reinterpret_cast<C*>(smem + off);     // [nx] coupling of line k to k-1
  off += (unsigned)(((nx + 1) & ~1) * 8);
  C* esh = reinterpret_cast<C*>(smem + off);     // [nx] coupling of line k to k+1
  off += (unsigned)(((nx + 1) & ~1) * 8);
  // complex64: [row tile][class][3] (offset within the stage, bit 31 transposed; input offset) of the row tile's tiles
  uint2* tiles = reinterpret_cast<uint2*>(smem + off);
  off += kSymTilesMax * 4 * 3 * 8;
  C* esc = reinterpret_cast<C*>(smem + off);           // [n16] the scaling of a point
  off += (unsigned)(n16 * 8);
  unsigned char* linef = smem + off;     // [nx] bit 0: grid line; 1, 2: owned in x (non-shifted, shifted); 3: source line
  off += (unsigned)((nx + 15) & ~15);
  DevSlot* sl = reinterpret_cast<DevSlot*>(smem + off);
  off += (unsigned)((sizeof(DevSlot) * R + 15) & ~size_t(15));
  SlotCoef* cf = reinterpret_cast<SlotCoef*>(smem + off);
  off += (unsigned)(sizeof(SlotCoef) * R);
  OutSlot* osl = reinterpret_cast<OutSlot*>(smem + off);

  const C* tr = reinterpret_cast<const C*>(a.traces);
  C* trw = reinterpret_cast<C*>(a.traces);
  const double2* x_in = a.x_ref ? *a.x_ref : a.x_in;   // the VOLUME input
  const unsigned char* fac = reinterpret_cast<const unsigned char*>(a.fac) + cl.fac_off * 8;
  C* scr = reinterpret_cast<C*>(a.scratch) + it.scratch_off;   // y_k / z_k
  // x_k: over y_k on one CTA per half (the lane that reads y_k writes x_k);
  // else in rows of its own, since another CTA may not have read y_k yet
  C* xscr = CL > 1 ? scr + (size_t)(nx + 1) * ny * R : scr;
  C* outs = reinterpret_cast<C*>(a.outs);
  const double2* px = a.prof + cl.prof_off;   // lo_x[nx], hi_x[nx], dg_x[nx], lo_y[ny], hi_y[ny], dg_y[ny], off_y[ny], e_y[ny]
  const double2* py = px + 3 * nx;

  // ---- set-up ----
  if (tid < R) {
    DevSlot s{};
    SlotCoef c{};
    if (tid < nslot) {
      s = a.slots[it.slot_begin + tid];
      if (s.kind == SK_DIR_X || s.kind == SK_CORNER) {
        c.c_oi_x = s.dx > 0 ? px[nx + s.xo] : px[s.xo];
        c.c_io_x = s.dx > 0 ? px[s.xi] : px[nx + s.xi];
      }
      if (s.kind == SK_DIR_Y || s.kind == SK_CORNER) {
        c.c_oi_y = s.dy > 0 ? py[ny + s.yo] : py[s.yo];
        c.c_io_y = s.dy > 0 ? py[s.yi] : py[ny + s.yi];
      }
    } else {
      s.kind = SK_NONE;
    }
    sl[tid] = s;
    cf[tid] = c;
  }
  if (tid >= 32 && tid - 32 < it.group_count) {
    // a slot's place in its group's sum, and the group's owned box and output
    const DevGroup G = a.groups[it.group_begin + tid - 32];
    const int gx = G.shift & 1, gy = (G.shift >> 1) & 1;
    OutSlot o;
    o.off = G.out_off;
    o.k0 = gx ? cl.ownx[1][0] : cl.ownx[0][0];
    o.k1 = gx ? cl.ownx[1][1] : cl.ownx[0][1];
    o.j0 = gy ? cl.owny[1][0] : cl.owny[0][0];
    o.j1 = gy ? cl.owny[1][1] : cl.owny[0][1];
    for (int r = 0; r < G.slot_count; ++r) {
      o.first = r == 0;
      o.last = r == G.slot_count - 1 && G.out_off >= 0;
      osl[G.slot_begin + r] = o;
    }
  }
  for (int k = tid; k < nx; k += blockDim.x) {
    linef[k] = (unsigned char)((is_line(cl.lox + k - a.p + 1, a.m, a.N) ? 1 : 0) |
                               (k >= cl.ownx[0][0] && k <= cl.ownx[0][1] ? 2 : 0) |
                               (k >= cl.ownx[1][0] && k <= cl.ownx[1][1] ? 4 : 0));
    wsh[k] = to_c(px[k], czero<C>());
    esh[k] = to_c(px[nx + k], czero<C>());
  }
  // byte offset within its chunk of the tile of (row tile w, source block s), bit 31: transposed
  auto tile_of = [&](int w, int s) -> unsigned {
    const int q = (w + s) & 3, hi = max(w, s), lo = min(w, s);
    const int head = q_first + ((q - q_first) & ~(cpc - 1));    // first class of its chunk
    return (unsigned)(symt.column[nb][q][lo] + ((hi - lo) >> 2) - symt.first[nb][head]) * kTileB |
           (s > w ? 0x80000000u : 0u);
  };
  if (!SPLIT) {
    for (int i = tid; i < nb * 12; i += blockDim.x) {
      const int w = i / 12, q = (i / 3) & 3, s = ((q - w) & 3) + 4 * (i % 3);
      if (s < nb && q >= q_first && q < q_first + NQ) tiles[i] = make_uint2(tile_of(w, s), (unsigned)(16 * s * XS * 8));
    }
  }
  for (int j = tid; j < n16; j += blockDim.x)
    esc[j] = to_c(j < ny ? py[4 * ny + j] : make_double2(1.0, 0.0), czero<C>());
  // the input's padding rows (and mma columns past the slots) stay zero: their
  // products with the tiles' padding must be finite
  for (unsigned i = tid; i < 2 * x_bytes / 16; i += blockDim.x)
    reinterpret_cast<uint4*>(smem + x_off)[i] = make_uint4(0u, 0u, 0u, 0u);
  if (tid == 0) {
    *abort_flag = 0;
    for (int i = 0; i < NS; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], (unsigned)NCW); }
    // one local arrive (with the expected bytes) per line; the partial sums
    // land by st.async and complete the transaction count
    mbar_init(&pready[0], 1);
    mbar_init(&pready[1], 1);
    mbar_init(exitb, (unsigned)(CLT * NCW));
    mbar_init(fwdb, (unsigned)(CL * NCW));
    mbar_init(xch, 1);
    mbar_expect_tx(xch, (unsigned)(ny * R * 8));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (tid < nslot && (sl[tid].kind == SK_DIR_X || sl[tid].kind == SK_CORNER)) {
    // (several slots may mark the same line: the same value)
    linef[sl[tid].xo] |= 8;
    linef[sl[tid].xi] |= 8;
  }
  __syncthreads();
  // every CTA's barriers are initialised before anyone arrives remotely
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");

  // ============================ producer ============================
  if (warp == 0) {
    if (lane < 2) {
      int idx = 0, slot = 0;
      unsigned phase = 1;                // parity of the empty phase to wait for (the first pass waits for none)
      bool stopped = false, first = true;
      const int nch = NQ / cpc;
      for (int li = 0; li < nline && !stopped; ++li) {
        const unsigned char* blk = fac + (size_t)line_k(li) * cl.blk * 8;
        for (int c = 0; c < nch; ++c, ++idx) {
          if ((idx & 1) == lane) {       // lanes 0 and 1 issue alternate chunks
            // (consumers release the stages in order, so the phase waited for
            // cannot be two behind)
            if (!first && !mbar_wait<false>(&empty[slot], phase, a.err, abort_flag, a.wait_cycles)) {
              stopped = true;
              break;
            }
            const unsigned t0 = symt.first[nb][q_first + c * cpc] * kTileB;
            const unsigned bytes = symt.first[nb][q_first + (c + 1) * cpc] * kTileB - t0;
            mbar_expect_tx(&full[slot], bytes);   // (no bytes: a class without tiles, in a small cell)
            if (bytes) bulk_g2s(smem + ring_off + (unsigned)slot * stage_bytes, blk + t0, bytes, &full[slot]);
          }
          if (++slot == NS) { slot = 0; phase ^= 1u; first = false; }
        }
      }
      // Wait (bounded by the limit alone) until the last copies this lane
      // issued have landed: after an abort the consumers stop waiting for
      // them, and no copy may write into shared memory after the CTA has left.
      for (int q = max(0, idx - NS); q < idx; ++q)
        if ((q & 1) == lane) mbar_wait<false>(&full[q % NS], (unsigned)((q / NS) & 1), a.err, nullptr, a.wait_cycles);
    }
    return;
  }

  // ============================ consumers ============================
  if (warp > NCW) return;                // idle warp (small cell)
  const int w = warp - 1;                // my 16 rows: tile w
  const int ct = (warp - 1) * 32 + lane;
  const int g = lane >> 2, t = lane & 3;           // split: mma fragment coordinates
  const int rho = lane & 15, h = lane >> 4;        // complex64: row, column parity
  const bool writer = w >= w_lo && w < w_hi;
  const int row0 = 16 * w + (SPLIT ? g : rho), slot0 = SPLIT ? t : (R > 1 ? h * RH : 0);
  auto row_of = [&](int e) { return row0 + (SPLIT ? 8 * (e & 1) : 0); };
  auto slot_of = [&](int e) { return slot0 + (SPLIT ? 4 * (e >> 1) : e); };
  // element e's offset from element 0 in a [row][slot] array
  auto step_of = [&](int e) { return SPLIT ? (e & 1) * 8 * R + (e >> 1) * 4 : e; };
  const int rs0 = row0 * R + slot0;
  // bit e: element e exists
  unsigned have = 0;
#pragma unroll
  for (int e = 0; e < NE; ++e)
    if (row_of(e) < ny && slot_of(e) < R && (SPLIT || R > 1 || h == 0)) have |= 1u << e;
  // the scaling of my rows' right-hand sides
  C ei[SPLIT ? 2 : 1];
#pragma unroll
  for (int q = 0; q < (SPLIT ? 2 : 1); ++q)
    ei[q] = to_c(crcp(row_of(q) < ny ? py[4 * ny + row_of(q)] : make_double2(1.0, 0.0)), czero<C>());
  // Byte offset of my accesses within a tile as it is (base_n) or transposed
  // (base_t).  complex64: of columns (rows) ch + CS i of my row (column) rho and,
  // with two rows per lane, of row rho ^ 8, each by XOR masks.  split: of my
  // ldmatrix row, the transposed tile with its off-diagonal 8 x 8 blocks exchanged.
  constexpr int TR = sym_rows(R), CS = 2 * TR, NI = 8 / TR;   // rows, column step, columns of a lane
  const int ch = lane >> (5 - TR);
  const unsigned base_n = SPLIT ? (unsigned)(lane * 16) : (unsigned)((ch * 16 + (rho ^ (4 * ch))) * 8);
  const unsigned base_t = SPLIT ? (unsigned)(((lane & 7) | ((lane & 8) << 1) | ((lane & 16) >> 1)) * 16)
                                : (unsigned)((rho * 16 + (SymTiles::swz(rho) ^ ch)) * 8);
  // split: my ldmatrix row of the input, n = lane mod 8 of (real plane, k 0-7),
  // (real, k 8-15), (imaginary, k 0-7), (imaginary, k 8-15): (re, im) of a slot
  // against the real plane, (im, re) against the imaginary one, whose products
  // are subtracted (re) and added (im) at the end
  const unsigned sb_row = ((((lane & 1) != 0) != (lane >= 16) ? RP : 0) + ((lane & 7) >> 1)) * kSplitRow + (lane & 8 ? 16u : 0u);
  // split: my row tile's tiles, class by class (3 source blocks each): offset
  // within the stage; bits: exists, transposed
  constexpr int ND = SPLIT ? 3 * NQ : 1;
  unsigned doff[ND], tmask = 0, tnmask = 0;
  if constexpr (SPLIT) {
#pragma unroll
    for (int i = 0; i < ND; ++i) {
      const int s = ((q_first + i / 3 - w) & 3) + 4 * (i % 3);
      doff[i] = 0;
      if (s < nb) {
        const unsigned d = tile_of(w, s);
        tmask |= 1u << i;
        if ((int)d < 0) tnmask |= 1u << i;
        doff[i] = (d & 0x7fffffffu) + ((int)d < 0 ? base_t : base_n);
      }
    }
  }

  // ---- right-hand sides, a line ahead ----
  // Volume (stage 1) and cell-vector slots: the raw double2 of the input;
  // trace slots: the trace value and its coefficient.  What depends on a load
  // is left to the use of the value, a line later.
  const bool vol = sl[0].kind == SK_VOLUME || sl[0].kind == SK_CELLVEC;
  // On an ordinary line an element of a trace slot takes c v[k] for k in its
  // range: its row is on the slot's outer or inner y-source line, and for an
  // L-sweep k is inside the x-source lines.  (PRE: kept per lane, up to 4
  // elements; else formed from the slot every line.)
  constexpr bool PRE = NE <= 4;
  unsigned rsel = 0;   // 2 bits per element: row on the outer (1) or inner (2) y-source line; volume: row in the window
  const C* bp[PRE ? NE : 1];
  C bc[PRE ? NE : 1];
  int bk[PRE ? NE : 1];                  // first line | one past the last << 16
#pragma unroll
  for (int e = 0; e < NE; ++e) {
    if constexpr (PRE) { bp[e] = tr; bc[e] = czero<C>(); bk[e] = 0; }
    if (!((have >> e) & 1)) continue;
    const DevSlot& s = sl[slot_of(e)];
    const int row = row_of(e);
    unsigned v = 0;
    if (s.kind == SK_VOLUME) {
      const int sy = (s.shift >> 1) & 1;
      v = row >= (sy ? cl.owny[1][0] : cl.owny[0][0]) && row <= (sy ? cl.owny[1][1] : cl.owny[0][1]) &&
          (int)is_line(cl.loy + row - a.p + 1, a.m, a.N) == sy;
    } else if (s.kind == SK_CELLVEC) {
      v = 1;
    } else if (s.kind == SK_DIR_Y || s.kind == SK_CORNER) {
      v = row == s.yo ? 1 : (row == s.yi ? 2 : 0);
      if constexpr (PRE) {
        if (v) {
          const C c = v == 1 ? to_c(cf[slot_of(e)].c_oi_y, czero<C>()) : cneg(to_c(cf[slot_of(e)].c_io_y, czero<C>()));
          bc[e] = cmul(c, ei[SPLIT ? (e & 1) : 0]);
          bp[e] = tr + (v == 1 ? s.in_ud1 : s.in_ud0);
          const int k0 = s.kind == SK_CORNER && s.dx > 0 ? s.xi + 1 : 0;
          const int k1 = s.kind == SK_CORNER && s.dx < 0 ? s.xi : nx;
          bk[e] = k0 | (k1 << 16);
        }
      }
    }
    rsel |= v << (2 * e);
  }
  float4 raw[NE];
  auto load_b = [&](int k, int fx) {
#pragma unroll
    for (int e = 0; e < NE; ++e) raw[e] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (vol) {
#pragma unroll
      for (int e = 0; e < NE; ++e) {
        if (((rsel >> (2 * e)) & 3) == 0) continue;
        const DevSlot& s = sl[slot_of(e)];
        const double2* p;
        if (s.kind == SK_VOLUME) {
          const int sx = s.shift & 1;
          if (!((fx >> (1 + sx)) & 1) || (fx & 1) != sx) continue;
          p = x_in + (long long)s.rhs * a.x_stride + (long long)(cl.lox + k) * a.n_dof + cl.loy + row_of(e);
        } else {
          p = a.x_in + (long long)s.rhs * a.x_stride + (long long)k * ny + row_of(e);
        }
        raw[e] = *reinterpret_cast<const float4*>(p);
      }
    } else if (fx & 8) {
      // a source line of some slot
#pragma unroll
      for (int e = 0; e < NE; ++e) {
        if (!((have >> e) & 1)) continue;
        const int r = slot_of(e);
        if (sl[r].kind == SK_NONE) continue;
        const C v = rhs_elem<float>(a, cl, sl[r], cf[r], tr, k, row_of(e)), c = ei[SPLIT ? (e & 1) : 0];
        raw[e] = make_float4(v.x, v.y, c.x, c.y);
      }
    } else if constexpr (PRE) {
#pragma unroll
      for (int e = 0; e < NE; ++e)
        if (k >= (bk[e] & 0xffff) && k < (bk[e] >> 16)) {
          const C v = bp[e][k];
          raw[e] = make_float4(v.x, v.y, bc[e].x, bc[e].y);
        }
    } else {
#pragma unroll
      for (int e = 0; e < NE; ++e) {
        const unsigned rs = (rsel >> (2 * e)) & 3;
        if (!rs) continue;
        const int r = slot_of(e);
        const DevSlot& s = sl[r];
        if (s.kind != SK_DIR_Y && (k - s.xi) * s.dx <= 0) continue;
        const C v = tr[(rs == 1 ? s.in_ud1 : s.in_ud0) + k];
        const C c = cmul(rs == 1 ? to_c(cf[r].c_oi_y, v) : cneg(to_c(cf[r].c_io_y, v)), ei[SPLIT ? (e & 1) : 0]);
        raw[e] = make_float4(v.x, v.y, c.x, c.y);
      }
    }
  };
  auto b_of = [&](int e) {
    if (vol) {
      double2 d;
      *reinterpret_cast<float4*>(&d) = raw[e];
      return cmul(to_c(d, czero<C>()), ei[SPLIT ? (e & 1) : 0]);
    }
    return cmul(make_float2(raw[e].z, raw[e].w), make_float2(raw[e].x, raw[e].y));
  };

  // ---- the line input ----
  // split: the row my address names of the four matrices of put_input: matrix lane / 8 (term, row half), row lane mod 8
  // (slot, part)
  const unsigned smem_a = saddr(smem);
  const unsigned st_row = (unsigned)((((lane >> 4) * 2 + (lane & 1)) * RP + ((lane >> 1) & 3)) * (int)kSplitRow + 32 * w +
                                     ((lane >> 3) & 1) * 16);
  auto put_input = [&](unsigned xb, const C (&v)[NE]) {
    if constexpr (SPLIT) {
      // [hi, lo][re, im][slot][point] bf16: a lane's words are (re, im) of a point
      // and slot, the fragment of an 8 x 8 matrix whose transpose has its rows there:
      // rows 0-7 and 8-15 of the hi words, then of the lo words, in one store
      // (16-bit stores, eight of a lane per 4 slots, took 2-3 % of a line: 8 x 8 cells of
      // 128^2 with 4 slots on 2 CTAs per half 6.84 -> 6.61 ms an apply)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        unsigned u[4];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int e = 2 * nt + i;
          const __nv_bfloat162 hb = __floats2bfloat162_rn(v[e].x, v[e].y);
          const __nv_bfloat162 lb = __floats2bfloat162_rn(v[e].x - __low2float(hb), v[e].y - __high2float(hb));
          const bool on = (have >> e) & 1;         // (padding stays zero)
          u[i] = on ? *reinterpret_cast<const unsigned*>(&hb) : 0u;
          u[2 + i] = on ? *reinterpret_cast<const unsigned*>(&lb) : 0u;
        }
        stsm4_t(smem_a + xb + st_row + (unsigned)(nt * 4) * kSplitRow, u);
      }
    } else {
      C* X = reinterpret_cast<C*>(smem + xb) + row0 * XS + slot0;
      if constexpr (V4) {
        if (have) {
#pragma unroll
          for (int e = 0; e < NE; e += 2)
            *reinterpret_cast<float4*>(X + e) = make_float4(v[e].x, v[e].y, v[e + 1].x, v[e + 1].y);
        }
      } else {
#pragma unroll
        for (int e = 0; e < NE; ++e)
          if ((have >> e) & 1) X[e] = v[e];
      }
    }
  };

  // ---- the exchange with the other CTAs of the half ----
  unsigned rq[CL > 1 ? CL - 1 : 1], rb[CL > 1 ? CL - 1 : 1];   // CTA me ^ d: my elements in its plane d - 1, its pready[0]
#pragma unroll
  for (int d = 1; d < CL; ++d) {
    rq[d - 1] = mapa(saddr(smem + q_off + (unsigned)(d - 1) * q_plane) + (unsigned)rs0 * 8u, rbase + (unsigned)(me ^ d));
    rb[d - 1] = mapa(saddr(pready), rbase + (unsigned)(me ^ d));
  }
  const unsigned line_bytes = (unsigned)((CL - 1) * ny * R * 8);
  if (CL > 1 && ct == 0) mbar_expect_tx(&pready[0], line_bytes);

  // waits by shared-memory address; the bounded wait only where the phase is not there yet
  const unsigned full_a = saddr(full), pready_a = saddr(pready), ring_a = smem_a + ring_off;
  auto phase_done = [](unsigned bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
  };
  // ---- one line: sums of my rows over every tile of the line ----
  unsigned fphase = 0;                   // the ring stage's parity
  unsigned par = 0, pphase = 0;          // exchange buffer of the line, its parity
  unsigned stage_a = ring_a, full_s = full_a;   // the current stage and its barrier
  const unsigned ring_end = ring_a + (unsigned)NS * stage_bytes;
  const unsigned cmask = (unsigned)(cpc - 1);
  auto line_product = [&](unsigned xb, bool more, C (&s)[NE]) {
    // arm the next line's barrier (peers' bytes may land before this; the
    // phase cannot complete without this arrive)
    if (CL > 1 && ct == 0 && more) mbar_expect_tx(&pready[par ^ 1u], line_bytes);
    C own[NE];
    // classes in turn: the chunk's wait at its first class, its release after the last
    auto enter = [&](int qi) {
      if ((qi & cmask) == 0 && !phase_done(full_s, fphase))
        mbar_wait<false>(full + (full_s - full_a) / 8, fphase, a.err, abort_flag, a.wait_cycles);
      return stage_a;
    };
    auto leave = [&](int qi) {
      if (((qi + 1) & cmask) == 0) {
        __syncwarp();
        if (lane == 0) mbar_arrive_at(full_s + kRingMax * 8u);   // the stage's empty barrier
        stage_a += stage_bytes;
        full_s += 8u;
        if (stage_a == ring_end) { stage_a = ring_a; full_s = full_a; fphase ^= 1u; }
      }
    };
    if constexpr (SPLIT) {
      float acc[2][NT][4];               // products with the real and the imaginary plane
#pragma unroll
      for (int p = 0; p < 2; ++p)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) acc[p][nt][0] = acc[p][nt][1] = acc[p][nt][2] = acc[p][nt][3] = 0.f;
      const unsigned xa = smem_a + xb + sb_row;
#pragma unroll
      for (int qi = 0; qi < NQ; ++qi) {
        const unsigned base = enter(qi), xq = xa + 32u * (unsigned)((q_first + qi - w) & 3);
#pragma unroll
        for (int n = 0; n < 3; ++n) {
          const int i = 3 * qi + n;
          if (4 * n >= nb) break;        // (uniform: the third and second blocks of small cells)
          // planes re hi, im hi, re lo, im lo; the loads predicated on the form of
          // the tile, and a block past the cell multiplies zeros: no branches
          unsigned e[4][4];
          const unsigned o = base + doff[i];
          ldsm4x4(e, o, (tmask >> i) & 1, (tnmask >> i) & 1);
#pragma unroll
          for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int q = 0; q < 2; ++q) {         // the input's hi, lo term
              unsigned b[4];
              ldsm4(b, xq + 128u * n + (unsigned)(q * 2 * RP + nt * 4) * kSplitRow);
#pragma unroll
              for (int p = 0; p < 2; ++p) {
                mma_bf16(acc[p][nt], e[p][0], e[p][1], e[p][2], e[p][3], b[2 * p], b[2 * p + 1]);
                mma_bf16(acc[p][nt], e[2 + p][0], e[2 + p][1], e[2 + p][2], e[2 + p][3], b[2 * p], b[2 * p + 1]);
              }
            }
        }
        leave(qi);
      }
#pragma unroll
      for (int e = 0; e < NE; ++e) {
        const int i = 2 * (e & 1), nt = e >> 1;
        own[e] = make_float2(acc[0][nt][i] - acc[1][nt][i], acc[0][nt][i + 1] + acc[1][nt][i + 1]);
      }
    } else {
      // sum[0]: my row; sum[1] (two rows per lane): row rho ^ 8, which is the row of lane ^ 8
      C sum[TR][R];
#pragma unroll
      for (int q = 0; q < TR; ++q)
#pragma unroll
        for (int r = 0; r < R; ++r) sum[q][r] = czero<C>();
      const unsigned char* xh = smem + xb + (unsigned)(ch * XS * 8);
#pragma unroll 1
      for (int qi = 0; qi < NQ; ++qi) {
        const uint2* tl = tiles + (w * 4 + q_first + qi) * 3;
        const int sb0 = (q_first + qi - w) & 3;
        const unsigned base = enter(qi);
#pragma unroll 1
        for (int sb = sb0; sb < nb; sb += 4, ++tl) {
          const uint2 d = *tl;
          const bool tn = (int)d.x < 0;
          // columns (rows) ch + CS i of the tile: XOR masks of the bits of i
          // (column CS i: 128 CS i bytes, rows swizzled by f(CS i)), and of row 8
          const unsigned o = base + (d.x & 0x7fffffffu) + (tn ? base_t : base_n);
          const unsigned m0 = TR == 2 ? (tn ? 32u : 512u | 8u) : (tn ? 16u : 256u | 64u);
          const unsigned m1 = TR == 2 ? (tn ? 64u : 1024u | 16u) : (tn ? 32u : 512u | 8u);
          const unsigned m2 = TR == 2 ? (tn ? 1024u | 16u : 64u) : (tn ? 64u : 1024u | 16u);
          const unsigned char* xp = xh + d.y;
          C v[8];                          // [row][column], or [column]
#pragma unroll
          for (int i = 0; i < 8; ++i) v[i] = lds_c(o ^ ((i & 1 ? m0 : 0u) ^ (i & 2 ? m1 : 0u) ^ (i & 4 ? m2 : 0u)));
#pragma unroll
          for (int i = 0; i < NI; ++i) {
            if constexpr (R == 1) {
              const C q = *reinterpret_cast<const C*>(xp + CS * i * 8);
#pragma unroll
              for (int u = 0; u < TR; ++u) cfma(sum[u][0], v[u * 4 + i], q);
            } else {
#pragma unroll
              for (int r = 0; r < R; r += 2) {
                const float4 q = *reinterpret_cast<const float4*>(xp + (CS * i * XS + r) * 8);
#pragma unroll
                for (int u = 0; u < TR; ++u) {
                  cfma(sum[u][r], v[u * 4 + i], make_float2(q.x, q.y));
                  cfma(sum[u][r + 1], v[u * 4 + i], make_float2(q.z, q.w));
                }
              }
            }
          }
        }
        leave(qi);
      }
      if constexpr (TR == 2) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          C got;
          got.x = __shfl_xor_sync(0xffffffffu, sum[1][r].x, 8);
          got.y = __shfl_xor_sync(0xffffffffu, sum[1][r].y, 8);
          sum[0][r] = cadd(sum[0][r], got);
        }
      }
#pragma unroll
      for (int e = 0; e < NE; ++e) {
        const C hi = sum[0][R > 1 ? RH + e : 0], lo = sum[0][R > 1 ? e : 0];
        const C keep = h && R > 1 ? hi : lo, give = h || R == 1 ? lo : hi;
        C got;
        got.x = __shfl_xor_sync(0xffffffffu, give.x, 16);
        got.y = __shfl_xor_sync(0xffffffffu, give.y, 16);
        own[e] = cadd(keep, got);
      }
    }
    if constexpr (CL > 1) {
      // my partial sums to every other CTA of the half, theirs from my buffer;
      // every CTA adds the same pairs
      const unsigned qo = par ? (CL - 1) * q_plane : 0u;
      const unsigned bo = par * 8u;
#pragma unroll
      for (int d = 1; d < CL; ++d) {
        if constexpr (V4) {
          if (have) {
#pragma unroll
            for (int e = 0; e < NE; e += 2) st_remote2(rq[d - 1] + qo + e * 8, own[e], own[e + 1], rb[d - 1] + bo);
          }
        } else {
#pragma unroll
          for (int e = 0; e < NE; ++e)
            if ((have >> e) & 1) st_remote(rq[d - 1] + qo + step_of(e) * 8, own[e], rb[d - 1] + bo);
        }
      }
      if (!phase_done(pready_a + par * 8u, pphase))
        mbar_wait<true>(&pready[par], pphase, a.err, abort_flag, a.wait_cycles);
      const C* src = reinterpret_cast<const C*>(smem + q_off + qo) + rs0;
      const int pl = n16 * R;
#pragma unroll
      for (int e = 0; e < NE; ++e) {
        s[e] = own[e];
        if ((have >> e) & 1) {
          s[e] = cadd(s[e], src[step_of(e)]);
          if constexpr (CL == 4) s[e] = cadd(s[e], cadd(src[pl + step_of(e)], src[2 * pl + step_of(e)]));
        }
      }
      pphase ^= par;
      par ^= 1u;
    } else {
#pragma unroll
      for (int e = 0; e < NE; ++e) s[e] = own[e];
    }
  };
  const int lstride = ny * R;
  auto store = [&](C* d, const C (&v)[NE]) {
    if (!writer) return;
    if constexpr (V4) {
      if (have) {
#pragma unroll
        for (int e = 0; e < NE; e += 2)
          *reinterpret_cast<float4*>(d + e) = make_float4(v[e].x, v[e].y, v[e + 1].x, v[e + 1].y);
      }
    } else {
#pragma unroll
      for (int e = 0; e < NE; ++e)
        if ((have >> e) & 1) d[step_of(e)] = v[e];
    }
  };

  C v[NE], s[NE];
  unsigned xb = x_off;
  const unsigned x_flip = x_off ^ (x_off + x_bytes);
  const bool warp_b = __any_sync(0xffffffffu, rsel != 0);   // my rows have right-hand sides on ordinary lines
  load_b(line_k(0), linef[line_k(0)]);
#pragma unroll
  for (int e = 0; e < NE; ++e) v[e] = b_of(e);
  put_input(xb, v);
  named_sync(1, NCT);

  // Lines in order; k runs away from my end of the cell and, after the middle
  // line, back.  A line's input, for the next line: b - (coupling) s (forward),
  // y_k - (coupling) s (backward); the coupling toward the next line of my
  // chain is w for the top half and e for the bottom half, backward the other.
  const int dk = half == 0 ? 1 : -1;
  int k = half == 0 ? 0 : nx - 1;
  C* sk = scr + (size_t)k * lstride + rs0;         // my elements of row k
  const ptrdiff_t xs_off = xscr - scr;
  const C* cpl = half == 0 ? wsh : esh;
#pragma unroll 1
  for (int li = 0; li < nline; ++li) {
    C cp = czero<C>();
    bool add = false;                              // raw holds what the input adds (uniform over the warp)
    if (li < nf) {
      const int kn = k + dk;             // (the middle line after my last)
      cp = cpl[kn];
      const int fx = linef[kn];
      add = warp_b || (fx & 8);
      if (add) load_b(kn, fx);
    } else if (li > nf) {
      cp = cpl[k];
      if constexpr (V4) {
#pragma unroll
        for (int e = 0; e < NE; e += 2) {
          const float4 q = have ? __ldcg(reinterpret_cast<const float4*>(sk + e)) : make_float4(0.f, 0.f, 0.f, 0.f);
          raw[e].x = q.x; raw[e].y = q.y; raw[e + 1].x = q.z; raw[e + 1].y = q.w;
        }
      } else {
#pragma unroll
        for (int e = 0; e < NE; ++e) {
          const C q = ((have >> e) & 1) ? __ldcg(sk + step_of(e)) : czero<C>();
          raw[e].x = q.x; raw[e].y = q.y;
        }
      }
    }
    line_product(xb, li + 1 < nline, s);
    xb ^= x_flip;
    if (li < nf) {
      // forward: y_k / z_k = s
#pragma unroll
      for (int e = 0; e < NE; ++e) v[e] = add ? b_of(e) : czero<C>();
      if (li + 1 < nf) {
#pragma unroll
        for (int e = 0; e < NE; ++e) cfms(v[e], cp, s[e]);
        put_input(xb, v);
        store(sk, s);
        k += dk;
        sk += dk * lstride;
      } else {
        store(sk, s);
        // the middle line's input b_m - w_m y_{m-1} - e_m z_{m+1}, formed in
        // the same order in both halves so that both compute the same x_m
        const unsigned partner = (unsigned)((1 - half) * CL + me);
        const unsigned pa = mapa(saddr(smem + p_off) + (unsigned)rs0 * 8u, partner), pb = mapa(saddr(xch), partner);
#pragma unroll
        for (int e = 0; e < NE; ++e)
          if ((have >> e) & 1) st_remote(pa + step_of(e) * 8, s[e], pb);
        if (CL > 1) {
          // my y_k are visible to the half once every warp of it has arrived
          __syncwarp();
          if (lane < CL) mbar_arrive_remote(fwdb, rbase + (unsigned)lane);
        }
        mbar_wait<true>(xch, 0u, a.err, abort_flag, a.wait_cycles);
        const C wm = wsh[mid], em = esh[mid];
        const C* P = reinterpret_cast<const C*>(smem + p_off) + rs0;
#pragma unroll
        for (int e = 0; e < NE; ++e) {
          const C oth = ((have >> e) & 1) ? P[step_of(e)] : czero<C>();
          cfms(v[e], wm, half == 0 ? s[e] : oth);
          cfms(v[e], em, half == 0 ? oth : s[e]);
        }
        put_input(xb, v);
      }
    } else if (li == nf) {
      // middle: x_m, the first backward input of both halves; k and sk are
      // already those of the first backward line
      put_input(xb, s);
      if (half == 0) store(sk + lstride + xs_off, s);
      if (CL > 1) mbar_wait<true>(fwdb, 0u, a.err, abort_flag, a.wait_cycles);
      cpl = half == 0 ? esh : wsh;
    } else {
      // backward: x_k = y_k - e_k (S_k^{-1} x_{k+1}) or z_k - w_k (T_k^{-1} x_{k-1})
#pragma unroll
      for (int e = 0; e < NE; ++e) {
        v[e] = make_float2(raw[e].x, raw[e].y);
        cfms(v[e], cp, s[e]);
      }
      put_input(xb, v);
      store(sk + xs_off, v);
      k -= dk;
      sk -= dk * lstride;
    }
    named_sync(1, NCT);
  }

  // ---- outputs of the solved item, from the x_k rows in scratch: owned DOFs
  // summed per (right-hand side, shift) group into the output
  // (DDCheckerboard::reduce, 744-772), the slots' outgoing trace lines into the
  // trace pool, and whole cell vectors for single-cell solves ----
  {
    const int jb = min(ny, 16 * w_lo), je = min(ny, 16 * w_hi), nJ = je - jb;   // my rows
    auto xat = [&](int k, int r, int j) { return xscr[((size_t)k * ny + j) * R + r]; };   // / e_j
    // points of my lines and rows that some shift owns, some at a time (their loads in flight
    // together), all slots of a point in one read
    constexpr int U = R <= 4 ? 4 : R <= 8 ? 2 : 1;
    const int ka = max(klo, min(cl.ownx[0][0], cl.ownx[1][0])), kb = min(khi, max(cl.ownx[0][1], cl.ownx[1][1]));
    const int ja = max(jb, min(cl.owny[0][0], cl.owny[1][0])), jw = min(je - 1, max(cl.owny[0][1], cl.owny[1][1])) - ja + 1;
    const int npt = (kb - ka + 1) * jw;
    if (it.group_count > 0 && jw > 0) {
      for (int e0 = ct; e0 < npt; e0 += U * NCT) {
        C x[U][R];
        int kk[U], jj[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int e = e0 + u * NCT;
          kk[u] = ka + e / jw;
          jj[u] = ja + e % jw;
          if (e >= npt) { kk[u] = -1; continue; }
          const C* p = xscr + ((size_t)kk[u] * ny + jj[u]) * R;
          if constexpr (R % 2 == 0) {
#pragma unroll
            for (int r = 0; r < R; r += 2) {
              const float4 q = *reinterpret_cast<const float4*>(p + r);
              x[u][r] = make_float2(q.x, q.y);
              x[u][r + 1] = make_float2(q.z, q.w);
            }
          } else {
            x[u][0] = p[0];
          }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (kk[u] < 0) continue;
          C sum = czero<C>();
          const C es = esc[jj[u]];
#pragma unroll
          for (int r = 0; r < R; ++r) {
            if (r >= nslot) break;
            const OutSlot& os = osl[r];
            sum = os.first ? x[u][r] : cadd(sum, x[u][r]);
            if (os.last && kk[u] >= os.k0 && kk[u] <= os.k1 && jj[u] >= os.j0 && jj[u] <= os.j1)
              red_add2(outs + os.off + (long long)(cl.lox + kk[u]) * a.n_dof + cl.loy + jj[u], cmul(sum, es));
          }
        }
      }
    }
    if (vol && sl[0].kind == SK_CELLVEC) {
      for (int r = 0; r < nslot; ++r)
        for (int e = ct; e < (khi - klo + 1) * nJ; e += NCT) {
          const int k = klo + e / nJ, j = jb + (e - (e / nJ) * nJ);
          a.x_out[(long long)sl[r].rhs * a.out_stride + (long long)k * ny + j] =
              to_c(cmul(xat(k, r, j), esc[j]), make_double2(0, 0));
        }
    } else {
      // a warp takes whole (slot, outgoing line) pairs, its loads in flight together
      for (int q = w; q < 8 * nslot; q += NCW) {
        const DevSlot& sr = sl[q >> 3];
        const int r = q >> 3, l = q & 3;
        const bool lr = (q & 4) == 0;
        if (l >= (lr ? sr.n_lr : sr.n_ud)) continue;
        // trace values; where lines cross, BL2TR overwrites trace0 entries
        // before they are added (DDCheckerboard.cpp:2520-2526)
        auto tval = [&](int k, int j) {
          if (sr.overwrite) {
            if (j == sr.yo) return tr[sr.in_ud0 + k];
            if (k == sr.xo) return tr[sr.in_lr0 + j];
          }
          return cmul(xat(k, r, j), esc[j]);
        };
        const int at = lr ? sr.lr_line[l] : sr.ud_line[l];
        const int p0 = lr ? jb : klo, p1 = lr ? je - 1 : khi;
        if (lr ? (at < klo || at > khi) : (at < jb || at >= je)) continue;
        C* dst = trw + (lr ? sr.lr_out[l] : sr.ud_out[l]);
        C tv[6];                             // a line of up to 192 points
#pragma unroll
        for (int u = 0; u < 6; ++u) {
          const int p = p0 + lane + 32 * u;
          if (p <= p1) tv[u] = lr ? tval(at, p) : tval(p, at);
        }
#pragma unroll
        for (int u = 0; u < 6; ++u) {
          const int p = p0 + lane + 32 * u;
          if (p <= p1) red_add2(dst + p, tv[u]);
        }
      }
    }
  }

  // nobody leaves while a peer may still write into its shared memory (waited
  // on even after an abort, bounded by the limit alone)
  __syncwarp();
  if (lane < CLT) mbar_arrive_remote(exitb, (unsigned)lane);
  mbar_wait<true>(exitb, 0u, a.err, nullptr, a.wait_cycles);
}

template <int CL, bool SPLIT>
__global__ void __launch_bounds__(32 * kSymWarps, 1) k_front_sym(FrontArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  const DevItem it = a.items[blockIdx.x / (2 * CL)];
  const DevCell cl = a.cells[it.cell];
  const int n = it.slot_count;
  if (n <= 1) sym_body<1, CL, SPLIT>(a, it, cl, smem);
  else if (n <= 2) sym_body<2, CL, SPLIT>(a, it, cl, smem);
  else if (n <= 4) sym_body<4, CL, SPLIT>(a, it, cl, smem);
  else if (n <= 8) sym_body<8, CL, SPLIT>(a, it, cl, smem);
  else if (n <= 12) sym_body<12, CL, SPLIT>(a, it, cl, smem);
  else sym_body<16, CL, SPLIT>(a, it, cl, smem);
}

}  // namespace

}  // namespace lsw
