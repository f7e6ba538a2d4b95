// Multi-RHS HMVM of plain plans on the FP64 matrix instruction: Y = H X for NR
// (2, 4 or 8) right-hand sides per pass, over the same planner layout as the
// single-vector kernels.
//
//   hmvm_dmma_kernel  one warp per team; the matrix streams through the warp's
//                     TMA ring as in hmvm_stream_kernel; the inputs of an item
//                     (its x or t columns, NR contiguous values each) come in
//                     pages, one page ahead, one bulk copy per segment.  Each
//                     step multiplies 4 columns of up to 32 rows by their 8
//                     inputs with one mma.m8n8k4.f64 per 8 rows.
//
// What bounds it and why this form.  With a lane per row on the FP64 units
// (hmvm_multi_kernel, which FP64 plans used before) every column cost a lane
// one matrix value and NR inputs from shared memory: 64 instructions per
// 16-byte vector of a tile, issued one in 5.5 cycles by each of 8 warps per SM,
// so the stages ran at 0.35 of the measured HBM rate with every pipe mostly
// idle.  The matrix instruction takes its operands spread over the lanes (one
// matrix and one input value each for 256 products), so a step of 4 columns is
// 9 loads and instructions.  tcgen05 has no FP64 kind; mma.sync is the only form
// of the FP64 matrix instruction.  It runs at the FP64 units' rate (measured 4
// cycles per SM, 64 products per cycle): 64 matrix bytes per cycle and SM
// against the 23 that HBM delivers, at any NR, so the stream stays the bound.
// What is left is latency per item (inputs, descriptors, outputs) that 12 warps
// per SM do not hide.
//
// FP32 plans: the matrix values come from ldmatrix in the operand's layout and
// are widened to FP64 in registers, as are the inputs, so products and sums are
// FP64 (error against FP64 2e-7 -> 4e-8).  A vector is a whole step there, so the
// FP64 pipe is busy for half of the row stage.  tf32 or 16-bit splits on the
// tensor cores would have been less exact than the FP32 sums they replaced.
//
// A team adds up the consecutive parts of a tile that it has (one page of inputs
// each), so only tiles that two teams share have partial sums.
//
// Measured, 8 right-hand sides, whole apply (V stage, row stage): N = 65,536 FP64
// sphere, 1.04 GB: 464 us (147, 295) -> 227 (75, 123: 5.5 TB/s); N = 100,003 FP32
// cube, 0.95 GB: 402 us (134, 237) -> 253 (84, 155: 3.9 TB/s).  m16n8k8 in place of
// four m8n8k4 changed nothing (251.3 to 250.6 us), nor did leaving out the
// conversions to FP64 (246): 12 warps waiting for dependent instructions (2.9 of 7
// cycles each) and for their ring are what is left.
#pragma once

#include "kernels_multi.cuh"

namespace hmvm {

// D += A B: A 8 x 4 (lane l: row l / 4, column l % 4), B 4 x 8 (lane l: row
// l % 4, column l / 4), D 8 x 8 (lane l: row l / 4, columns 2 (l % 4) + {0, 1}).
__device__ __forceinline__ void dmma884(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

// The 32-bit words of up to 32 rows of 16 bytes: lane l gives the address of row
// l and gets, per block of 8 rows, word l % 4 of row l / 4 (the A operand's layout).
template <int NRB>
__device__ __forceinline__ void ldmatrix_words(uint32_t (&w)[4], uint32_t addr) {
  if constexpr (NRB == 1)
    asm volatile("ldmatrix.sync.aligned.m8n8.x1.shared.b16 {%0}, [%1];" : "=r"(w[0]) : "r"(addr) : "memory");
  else if constexpr (NRB == 2)
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0, %1}, [%2];" : "=r"(w[0]), "=r"(w[1]) : "r"(addr) : "memory");
  else
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3])
                 : "r"(addr)
                 : "memory");
}

template <int WPB, int S, int CHUNK>
constexpr int dmma_min_blocks() {
  constexpr int by_smem = (227 * 1024) / (dmma_smem_bytes(MultiCfg{WPB, S, CHUNK}) + 1024);
  return by_smem > 0 ? by_smem : 1;
}

// The body of hmvm_dmma_kernel for block bid of the launch (a batch launch runs
// several plans' bodies, each over its own range of blocks).  CHECK: every
// input range and output row is checked against the buffers' lengths; a miss
// records error 3 and is skipped.  NRC: the pass width, or 0 for one that is only
// known at run time (nr; a batch's parts differ, and one body per width made its
// kernel outgrow the instruction cache: 6 of 11 cycles per instruction waiting
// for it).
template <typename T, int WPB, int S, int CHUNK, int NRC, bool VST, bool CHECK = false>
__device__ __forceinline__ void dmma_body(const MultiArgs& a, int bid, int nr = NRC) {
  constexpr uint32_t RING = (uint32_t)S * CHUNK;
  constexpr uint32_t RSTRIDE = RING + kDmmaRingPad;  // the ring and the copy of its first bytes
  constexpr int VN = 16 / (int)sizeof(T);  // columns per 16-byte vector
  constexpr int SV = 4 / VN;               // vectors per step of 4 columns
  constexpr int B = 8;                     // vectors per batch
  constexpr int NS = B / SV;               // steps per batch
  const int NR = NRC > 0 ? NRC : nr;       // 2 (FP64 only), 4 or 8
  const int ES = NR * (int)sizeof(T);      // input bytes per column
  const int PVL = (NR == 2 ? 3 : NR == 4 ? 2 : 1) + 4;  // log2 of the vectors per page of inputs
  const int PV = 1 << PVL;
  using T2 = typename std::conditional<std::is_same<T, double>::value, double2, float2>::type;
  static_assert((RING & (RING - 1)) == 0, "ring size must be a power of two");
  static_assert(CHUNK % 16 == 0 && CHUNK >= 512, "bulk copies move multiples of 16 bytes");
  static_assert(B * 32 * 16 <= (S - 1) * CHUNK, "ring too small for one batch");
  static_assert(NRC == 0 || NRC == 2 || NRC == 4 || NRC == 8, "one block of 8 result columns");
  static_assert(kDmmaPageBytes == 4096, "pages of 4096 / (16 NR) vectors, a whole number of batches");
  extern __shared__ __align__(128) unsigned char smem[];

  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int team = bid * WPB + warp;
  if (team >= a.nteams) return;
  const int tb = a.team_begin[team], te = a.team_begin[team + 1];
  if (tb >= te) return;
  unsigned char* ring = smem + (size_t)warp * RSTRIDE;
  unsigned char* zbase = smem + (size_t)WPB * RSTRIDE + (size_t)warp * 2 * kDmmaPageBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + (size_t)WPB * (RSTRIDE + 2 * kDmmaPageBytes)) + warp * (S + 2);
  uint64_t* zbars = bars + S;

  const hmvm_tile_desc* __restrict__ tiles = a.tiles;
  const hmvm_seg_desc* __restrict__ segs = a.segs;
  const T* __restrict__ xin = std::is_same<T, double>::value ? reinterpret_cast<const T*>(a.x64)
                                                             : reinterpret_cast<const T*>(a.x32);
  const hmvm_tile_desc dzero = {0, 0, 0, 0, 0, 1, 0, 0};
  const hmvm_seg_desc szero = {0, 0};

  hmvm_tile_desc cur = tiles[tb];
  const int64_t vbase = cur.data_off;
  const hmvm_tile_desc tl = tiles[te - 1];
  const int64_t total64 = (tl.data_off + (int64_t)tl.nvec * tl.nrows - vbase) * 16;
  if (total64 >= (int64_t)1 << 31) {
    if (lane == 0) atomicExch(a.err, 2);
    return;
  }
  const uint32_t total = (uint32_t)total64;
  const char* gsrc = static_cast<const char*>(a.data) + vbase * 16;
  const uint32_t nchunks = (total + CHUNK - 1) / CHUNK;
  if (lane == 0) {
#pragma unroll
    for (int s = 0; s < S + 2; s++) mbar_init(&bars[s], 1);
    fence_mbar_init();
  }
  __syncwarp();
  // Lane 0 only: start the copy of chunk q into slot q % S (the first bytes of
  // slot 0 also behind the ring's end, so that a vector that wraps around can
  // be read in one piece), and bring the chunk after it into L2.
  auto issue = [&](uint32_t q) {
    const uint32_t off = q * (uint32_t)CHUNK;
    const uint32_t bytes = min((uint32_t)CHUNK, total - off);
    const uint32_t again = q % S == 0 ? min((uint32_t)kDmmaRingPad, bytes) : 0;
    uint64_t* bar = &bars[q % S];
    mbar_expect_tx(bar, bytes + again);
    bulk_g2s(ring + (q % S) * CHUNK, gsrc + off, bytes, bar);
    if (again > 0) bulk_g2s(ring + RING, gsrc + off, again, bar);
    if (q + 1 < nchunks) bulk_prefetch_l2(gsrc + off + CHUNK, min((uint32_t)CHUNK, total - off - CHUNK));
  };
  if (lane == 0)
    for (uint32_t q = 0; q < min((uint32_t)S, nchunks); q++) issue(q);

  // Page pg of an item's inputs (columns [pg * PV * VN, ...) of its padded
  // segments) into buffer b: lane j copies its part of segment j (contiguous)
  // onto the buffer's mbarrier; the padding of a segment to whole vectors is
  // zeroed with plain stores (its matrix entries are zero, and what follows
  // the segment in x need not be finite).  `from` is the group of 32 segments
  // that the page starts in, and is left at the one it ends in, where the next
  // page goes on.  (A scan of all segments for each page made a run of hundreds
  // of them, 1 to 2 columns each, 1.3 to 2.4 times as long.)
  auto gather = [&](int seg_begin, int nseg, const hmvm_seg_desc& sreg, int sfirst, int pg, int b, int& from) {
    unsigned char* zb = zbase + b * kDmmaPageBytes;
    uint64_t* zbar = &zbars[b];
    const int lo = pg * (PV * VN), hi = lo + PV * VN;
    fence_proxy_async();  // the buffer's earlier generic reads before the async writes
    for (;; from += 32) {
      hmvm_seg_desc my = sreg;
      int first = sfirst;
      if (from > 0) {
        const bool has = from + lane < nseg;
        my = has ? segs[seg_begin + from + lane] : szero;
        first = has ? a.seg_first[seg_begin + from + lane] : 0;
      }
      const int nc = my.ncols, ncp = (nc + VN - 1) / VN * VN;
      const bool from_t = my.src < 0;
      const int p0 = max(first, lo), p1 = min(first + ncp, hi);  // the segment's part of this page
      int copied = max(0, min(first + nc, hi) - p0);
      const int64_t src = (int64_t)((from_t ? (my.src & 0x7fffffff) : my.src) + p0 - first) * NR;
      if constexpr (CHECK) {
        if (p1 > p0 && src + (int64_t)(p1 - p0) * NR > (from_t ? a.tcap : a.xcap)) {
          atomicExch(a.err, 3);
          copied = 0;
        }
      }
      const uint32_t gbytes = __reduce_add_sync(0xffffffffu, (uint32_t)(copied * ES));
      if (lane == 0 && gbytes > 0) mbar_expect_tx_only(zbar, gbytes);
      __syncwarp();
      unsigned char* dst = zb + (p0 - lo) * ES;
      if (copied > 0) bulk_g2s(dst, (from_t ? static_cast<const T*>(a.t) : xin) + src, (uint32_t)(copied * ES), zbar);
      for (int z = copied; z < p1 - p0; z++)
        for (int r = 0; r < ES; r += 16) *reinterpret_cast<uint4*>(dst + z * ES + r) = make_uint4(0, 0, 0, 0);
      if (from + 32 >= nseg || __shfl_sync(0xffffffffu, first + ncp, 31) >= hi) break;
    }
    if (lane == 0) mbar_arrive(zbar);
  };
  auto out_slot = [&](const hmvm_tile_desc& d) {
    if constexpr (VST) return (d.mode == 1 && lane < d.nrows) ? a.out_idx[d.out_base + lane] : 0;
    else return 0;
  };

  auto seg_of = [&](const hmvm_tile_desc& d) { return lane < d.nseg ? segs[d.seg_begin + lane] : szero; };
  auto first_of = [&](const hmvm_tile_desc& d) { return lane < d.nseg ? a.seg_first[d.seg_begin + lane] : 0; };
  hmvm_seg_desc cur_seg = seg_of(cur);
  int cur_first = first_of(cur);
  int seg_from = 0;  // where the next page of the item whose inputs are being fetched starts
  gather(cur.seg_begin, cur.nseg, cur_seg, cur_first, 0, 0, seg_from);
  int cur_oidx = out_slot(cur);
  hmvm_tile_desc nxt = tb + 1 < te ? tiles[tb + 1] : dzero;
  hmvm_seg_desc nxt_seg = seg_of(nxt);
  int nxt_first = first_of(nxt), nxt_oidx = out_slot(nxt);
  hmvm_tile_desc nn = tb + 2 < te ? tiles[tb + 2] : dzero;

  const int kq = lane & 3, nq = lane >> 2;  // the lane's column within a step and its input / row of a block
  const bool has_z = NR == 8 || nq < NR;
  uint32_t q_ready = 0, q_rel = 0;
  uint32_t kp = 0, gathered = 1;  // pages processed and started
  bool failed = false;
  for (int ti = tb; ti < te && !failed; ++ti) {
    // loads for two items ahead; they land while this item runs
    const hmvm_seg_desc nn_seg = seg_of(nn);
    const int nn_first = first_of(nn), nn_oidx = out_slot(nn);
    const hmvm_tile_desc nnn = ti + 3 < te ? tiles[ti + 3] : dzero;

    const int R = cur.nrows, nvt = cur.nvec;
    const uint32_t rstride = (uint32_t)R * 16;
    uint32_t o = (uint32_t)((cur.data_off - vbase) * 16);
    // the lane's place within a step (FP64: 8 bytes of row nq of the step's vector
    // kq / 2; FP32: the 16-byte row that the lane addresses for ldmatrix)
    const uint32_t lane_vec = sizeof(T) == 8 ? (uint32_t)(kq >> 1) * rstride : 0u;
    const unsigned char* lane_ring = ring + (sizeof(T) == 8 ? nq * 16 + (kq & 1) * 8 : lane * 16);
    // Sums of the page and of the item: pages are added up in order, which keeps
    // the chains of additions short.
    double acc[4][2], sum[4][2];
#pragma unroll
    for (int rb = 0; rb < 4; rb++) acc[rb][0] = acc[rb][1] = sum[rb][0] = sum[rb][1] = 0.0;
    // Vectors [v0, v1) of the item, NRB blocks of 8 rows.  Rows past R of the
    // last block read ring bytes of other rows (always inside the ring); a row
    // of the matrix operand only reaches its own row of the result, which is
    // not stored.
    auto run = [&](auto tag, int v0, int v1, const unsigned char* zpage) -> bool {
      constexpr int NRB = decltype(tag)::value;
      const T* zl = reinterpret_cast<const T*>(zpage) + kq * NR + (has_z ? nq : 0);
      for (int v = v0; v < v1; v += B, zl += B * VN * NR) {
        const int nb = min(B, v1 - v);
        const uint32_t o_end = o + (uint32_t)nb * rstride;
        if (o >= (q_rel + 1) * (uint32_t)CHUNK) {  // release the slots the warp has moved past
          const uint32_t qf = o / CHUNK;
          __syncwarp();
          if (lane == 0) {
            fence_proxy_async();
            for (uint32_t q = q_rel; q < qf; q++)
              if (q + S < nchunks) issue(q + S);
          }
          q_rel = qf;
        }
        if (o_end > q_ready * (uint32_t)CHUNK) {  // wait for the batch's chunks
          const uint32_t ql = (o_end - 1) / CHUNK;
          while (q_ready <= ql) {
            if (!warp_wait(&bars[q_ready % S], (q_ready / S) & 1)) return false;
            q_ready++;
          }
        }
        const uint32_t ol = o + lane_vec;
        double m[NS][NRB], z[NS];
        auto load = [&](int s, double (&ms)[NRB], double& zs) {
          zs = has_z ? (double)zl[s * 4 * NR] : 0.0;
          const unsigned char* rp = lane_ring + ((ol + (uint32_t)(s * SV) * rstride) & (RING - 1));
          if constexpr (sizeof(T) == 8) {
#pragma unroll
            for (int rb = 0; rb < NRB; rb++) ms[rb] = *reinterpret_cast<const double*>(rp + rb * 128);
          } else {
            uint32_t w[4];
            ldmatrix_words<NRB>(w, smem_u32(rp));
#pragma unroll
            for (int rb = 0; rb < NRB; rb++) ms[rb] = (double)__uint_as_float(w[rb]);
          }
        };
        if (nb == B) {
#pragma unroll
          for (int s = 0; s < NS; s++) load(s, m[s], z[s]);
#pragma unroll
          for (int s = 0; s < NS; s++)
#pragma unroll
            for (int rb = 0; rb < NRB; rb++) dmma884(acc[rb], m[s][rb], z[s]);
        } else {
#pragma unroll 1
          for (int s = 0; s * SV < nb; s++) {
            load(s, m[0], z[0]);
            if (SV == 2 && s * SV + (kq >> 1) >= nb) {  // an odd last FP64 vector is half a step
              z[0] = 0.0;
#pragma unroll
              for (int rb = 0; rb < NRB; rb++) m[0][rb] = 0.0;
            }
#pragma unroll
            for (int rb = 0; rb < NRB; rb++) dmma884(acc[rb], m[0][rb], z[0]);
          }
        }
        o = o_end;
      }
      return true;
    };
    const int npg = max(1, (nvt + PV - 1) >> PVL);
    for (int pg = 0; pg < npg; pg++, kp++) {
      __syncwarp();  // every lane is done with the page the next gather overwrites
      const uint32_t nbuf = (kp + 1) & 1;
      const bool more = pg + 1 < npg;
      if (more || ti + 1 < te) {
        if (!more) seg_from = 0;
        const hmvm_seg_desc gs = {more ? cur_seg.src : nxt_seg.src, more ? cur_seg.ncols : nxt_seg.ncols};
        gather(more ? cur.seg_begin : nxt.seg_begin, more ? cur.nseg : nxt.nseg, gs, more ? cur_first : nxt_first,
               more ? pg + 1 : 0, nbuf, seg_from);
        gathered++;
      }
      if (!warp_wait(&zbars[kp & 1], (kp >> 1) & 1)) {
        failed = true;
        break;
      }
      __syncwarp();  // and the zeroed padding
      const unsigned char* zpage = zbase + (kp & 1) * kDmmaPageBytes;
      const int v0 = pg * PV, v1 = min(nvt, v0 + PV);
      bool ok;
      switch ((R + 7) >> 3) {
        case 1: ok = run(TypeTag<1>{}, v0, v1, zpage); break;
        case 2: ok = run(TypeTag<2>{}, v0, v1, zpage); break;
        case 3: ok = run(TypeTag<3>{}, v0, v1, zpage); break;
        default: ok = run(TypeTag<4>{}, v0, v1, zpage); break;
      }
      if (!ok) {
        failed = true;
        break;
      }
#pragma unroll
      for (int rb = 0; rb < 4; rb++)
#pragma unroll
        for (int i = 0; i < 2; i++) {
          sum[rb][i] += acc[rb][i];
          acc[rb][i] = 0.0;
        }
    }
    if (failed) break;
    uint32_t row_ok = 0xffffffffu;  // rows whose outputs lie inside their buffer
    if constexpr (CHECK) {
      const int64_t hi = VST ? (cur.mode == 1 ? ((int64_t)cur_oidx + 1) * NR : ((int64_t)cur.out_base + R) * NR)
                             : (cur.mode == 0 ? (int64_t)cur.out_base + R + (int64_t)(NR - 1) * a.ldy
                                              : ((int64_t)cur.out_base + R) * NR);
      const int64_t cap = VST ? (cur.mode == 1 ? a.tcap : a.pcap) : (cur.mode == 0 ? a.ycap : a.pcap);
      row_ok = __ballot_sync(0xffffffffu, cur_oidx >= 0 && cur.out_base >= 0 && hi <= cap);
      if (row_ok != 0xffffffffu && lane == 0) atomicExch(a.err, 3);
    }
    // Lane l holds rows 8 rb + l / 4, right-hand sides 2 (l % 4) + {0, 1}.
#pragma unroll
    for (int rb = 0; rb < 4; rb++) {
      const int row = 8 * rb + nq, r = 2 * kq;
      const int slot = VST ? __shfl_sync(0xffffffffu, cur_oidx, row) : 0;
      if (row < R && r < NR && (!CHECK || (row_ok >> row & 1))) {
        T2 val;
        val.x = (T)sum[rb][0];
        val.y = (T)sum[rb][1];
        if (VST && cur.mode == 1) {
          *reinterpret_cast<T2*>(static_cast<T*>(a.t) + (int64_t)slot * NR + r) = val;
        } else if (!VST && cur.mode == 0) {
          T* y = static_cast<T*>(a.y) + cur.out_base + row + r * a.ldy;
          if (r < a.nr) y[0] = val.x;
          if (r + 1 < a.nr) y[a.ldy] = val.y;
        } else {
          *reinterpret_cast<T2*>(static_cast<T*>(a.p) + (int64_t)(cur.out_base + row) * NR + r) = val;
        }
      }
    }
    cur = nxt;
    cur_seg = nxt_seg;
    cur_first = nxt_first;
    cur_oidx = nxt_oidx;
    nxt = nn;
    nxt_seg = nn_seg;
    nxt_first = nn_first;
    nxt_oidx = nn_oidx;
    nn = nnn;
  }
  if (failed) {
    // Let every copy still in flight land before the CTA's shared memory goes away.
    const uint32_t issued = min(nchunks, q_rel + (uint32_t)S);
    for (uint32_t q = q_ready; q < issued; q++) warp_wait(&bars[q % S], (q / S) & 1);
    for (uint32_t i = kp; i < gathered; i++) warp_wait(&zbars[i & 1], (i >> 1) & 1);
    if (lane == 0) atomicExch(a.err, 1);
  }
}

template <typename T, int WPB, int S, int CHUNK, int NR, bool VST>
__global__ void __launch_bounds__(32 * WPB, (dmma_min_blocks<WPB, S, CHUNK>())) hmvm_dmma_kernel(MultiArgs a) {
  dmma_body<T, WPB, S, CHUNK, NR, VST>(a, (int)blockIdx.x);
}

}  // namespace hmvm
