// SELL-32 storage of the level matrices for the solve (sm_100a).
//
// The assembled matrix stays in the host's CSR pattern (that is what the
// slot map scatters into and what pmg_get_matrix returns).  For the solve
// every level also keeps a sliced-ELLPACK copy built once per pattern:
//
//   * rows are grouped by SSOR colour (Dirichlet rows form a last group),
//     sorted inside a group by decreasing length (ties: increasing row), and
//     cut into slices of 32 rows; a group is padded with empty rows to a
//     multiple of 32, so every colour owns a whole number of slices;
//   * slice s stores its 32 rows column-major in three parts: the entries of
//     lower colours, the diagonal (one step), the entries of higher colours,
//     each part as long as the slice's longest: entry j of lane l sits at
//     slice_ptr[s] + 32 j + l, so a warp reads 128 contiguous bytes (FP32) per
//     step; padding has value 0 and a valid column, so no masking is needed.
//     A product walks all steps; a Gauss-Seidel sweep needs one side of the
//     diagonal only, see k_sell_gs.
//
// A block of SELL_K warps owns one slice (each warp takes every SELL_K-th
// column step of the 32 rows), so every row keeps several independent
// load chains in flight; the CSR kernels with a W-lane group per row stall
// on the row pointer of every row.  Vectors stay in the host's dof
// numbering: the kernels gather x through L2 and write each result row once.
//
// An SSOR step runs in phases of several colours (sell_ssor): the part of a
// phase's rows that comes from outside is a product over the whole GPU, the
// colours of the phase then follow each other inside one CTA per block of
// rows.  A pattern whose phases do not fall into blocks takes one launch per
// colour and direction.  All launches are captured in the V-cycle's CUDA graph
// and chained with programmatic dependent launch.
#include "pmg_internal.h"
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>

namespace pmg {

// --------------------------------------------------------------- phases and blocks
// A phase is a range of consecutive colours.  Its rows are coupled among each
// other only inside the connected components (blocks) of the phase's part of
// the pattern, so within a phase every block can go through the colours on its
// own.  The lattice colourings have such phases: with 27 colours (3 x 3 x 3
// residues of the node indices) nine consecutive ones lie in planes three
// apart, with 8 colours four lie in planes two apart, and no entry joins two of
// them.  For any other pattern and colouring the components are simply looked
// at: a pattern whose phases hang together gets no blocks.
__global__ void k_cc_init(int n, int *parent) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) parent[i] = i;
}
__device__ __forceinline__ int cc_find(int *parent, int i) {
  int p = ((volatile int *)parent)[i];
  while (p != i) {
    const int q = ((volatile int *)parent)[p];
    if (q != p) atomicCAS(parent + i, p, q);  // path halving; losing the race does no harm
    i = p;
    p = q;
  }
  return i;
}
// union of the two ends of every entry inside a phase (a root only ever gets a
// smaller parent, so the trees have no cycles and every loop ends)
__global__ void k_cc_unite(int Na, const int *__restrict__ rp, const int *__restrict__ kc,
                           const int *__restrict__ colour, const int *__restrict__ phase, int *parent) {
  const int lane = threadIdx.x & 31;
  for (int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < Na; r += (gridDim.x * blockDim.x) >> 5)
    for (int k = rp[r] + lane; k < rp[r + 1]; k += 32) {
      const int c = kc[k];
      if (c >= Na || c == r || phase[colour[c]] != phase[colour[r]]) continue;
      int a = cc_find(parent, r), b = cc_find(parent, c);
      while (a != b) {
        if (a < b) { const int t = a; a = b; b = t; }
        const int old = atomicCAS(parent + a, a, b);
        if (old == a) break;
        a = cc_find(parent, old);
        b = cc_find(parent, b);
      }
    }
}
// (and the number of components of every phase)
__global__ void k_cc_flatten(int n, const int *__restrict__ colour, const int *__restrict__ phase, int *parent,
                             int *count) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int root = cc_find(parent, i);
  parent[i] = root;
  if (root == i) atomicAdd(count + phase[colour[i]], 1);
}

// a block's iterate sits in shared memory, addressed by 16-bit slots
constexpr size_t BLK_SMEM = 224 * 1024;
constexpr int BLK_MAX_COLOURS = 64;
constexpr int BLK_TASK = 16;  // bytes per task kept beside it

// Phases and blocks of a level: phase boundaries into L.blk_col (empty: none),
// block of every active row into blk.  About the cube root of the number of
// colours as the number of phases first (27 -> 3, 8 -> 2), then finer ones.
// d_colour: the colours on the device; d_phase, d_parent, d_count: device scratch of
// N + colours ints each.  slices: per phase those of each block.
static int find_blocks(Handle &h, Level &L, const std::vector<int> &colour, std::vector<int> &blk,
                       std::vector<std::vector<int>> &slices, const int *d_colour, int *d_phase, int *d_parent,
                       int *d_count) {
  const int N = L.N, Na = L.Na, nc = (int)L.rcolor_ptr.size() - 1;
  L.blk_col.clear();
  if (N <= CC_BLOCK_ROWS || nc < 3) return PMG_OK;
  const int s0 = std::max(2, (int)(cbrt((double)nc) + 0.5));
  std::vector<int> label;
  for (int S : {s0, s0 + 1, s0 * s0}) {
    if (S >= nc) break;
    std::vector<int> bound(S + 1);
    for (int p = 0; p <= S; p++) bound[p] = (int)((long)p * nc / S);
    // (the hops are counted in fixed arrays; and the tables below hold a number per
    // block and colour, which stays within 64 per row this way)
    if ((nc + S - 1) / S > BLK_MAX_COLOURS) continue;
    std::vector<int> phase_of(nc + 1, S);
    for (int p = 0; p < S; p++)
      for (int c = bound[p]; c < bound[p + 1]; c++) phase_of[c] = p;
    PMG_CUDA(cudaMemcpyAsync(d_phase, phase_of.data(), sizeof(int) * (nc + 1), cudaMemcpyHostToDevice, h.stream));
    PMG_CUDA(cudaMemsetAsync(d_count, 0, sizeof(int) * S, h.stream));
    k_cc_init<<<(Na + 255) / 256, 256, 0, h.stream>>>(Na, d_parent);
    k_cc_unite<<<h.num_sms * 8, 256, 0, h.stream>>>(Na, L.rowptr.p, L.kcol.p, d_colour, d_phase, d_parent);
    k_cc_flatten<<<(Na + 255) / 256, 256, 0, h.stream>>>(Na, d_colour, d_phase, d_parent, d_count);
    count_launches(3);
    PMG_CUDA(cudaGetLastError());
    std::vector<int> n(S, 0);
    PMG_CUDA(cudaMemcpyAsync(n.data(), d_count, sizeof(int) * S, cudaMemcpyDeviceToHost, h.stream));
    PMG_CUDA(cudaStreamSynchronize(h.stream));
    bool ok = true;
    for (int p = 0; p < S; p++) ok = ok && n[p] >= 4 && n[p] <= 65535;
    if (!ok) continue;
    label.resize(Na);
    PMG_CUDA(cudaMemcpyAsync(label.data(), d_parent, sizeof(int) * Na, cudaMemcpyDeviceToHost, h.stream));
    PMG_CUDA(cudaStreamSynchronize(h.stream));
    // number the blocks of each phase by their first rows; rows per block and colour
    std::fill(n.begin(), n.end(), 0);
    blk.assign(Na, -1);
    for (int r = 0; r < Na; r++)
      if (label[r] == r) blk[r] = n[phase_of[colour[r]]]++;
    std::vector<std::vector<int>> rows(S);
    for (int p = 0; p < S; p++) rows[p].assign((size_t)n[p] * (bound[p + 1] - bound[p]), 0);
    for (int r = 0; r < Na; r++) {
      const int p = phase_of[colour[r]];
      blk[r] = blk[label[r]];
      rows[p][(size_t)blk[r] * (bound[p + 1] - bound[p]) + colour[r] - bound[p]]++;
    }
    // a block's slots (rows padded to slices) fit shared memory in FP32 at
    // least, and the padding does not outweigh the rows
    size_t all = 0, largest = 0;
    slices.assign(S, {});
    for (int p = 0; p < S; p++) {
      const int w = bound[p + 1] - bound[p];
      slices[p].assign(n[p], 0);
      for (int b = 0; b < n[p]; b++) {
        for (int c = 0; c < w; c++) slices[p][b] += (rows[p][(size_t)b * w + c] + 31) / 32;
        const size_t slots = (size_t)slices[p][b] * 32;
        all += slots;
        largest = std::max(largest, slots);
      }
    }
    if (largest > 65535 || largest * sizeof(float) + largest / 32 * BLK_TASK > BLK_SMEM || all > 1.6 * Na) continue;
    L.blk_col = bound;
    L.blk_n = n;
    return PMG_OK;
  }
  return PMG_OK;
}

// Whether an SSOR step by blocks is the faster one, per precision: the time of a
// step's colour launches less that of its products and block sweeps, in us.  A block
// is swept by one CTA, so what counts is the largest one of a phase, or all of them
// and a start-up each where there are more than SMs.  The model is fitted to steps
// on the levels of Q1, Q2, P2 and non-conforming hierarchies of 5 k to 2.1 M rows and
// on slabs of 33^2 to 201^2 x 9 to 257 nodes (148 SMs): a launch 2.7 us; entries read
// by the whole GPU 0.4 / 0.2 us per MB (FP32 / FP64; the ones inside blocks are read
// by a few SMs and are in their terms); a block's slice 0.018 / 0.036 us and 0.009 /
// 0.016 us for every chunk of four inside entries, per pass; a block beyond the first
// 148 3.6 us.  It has the sign of the measured difference in 107 of 114 cases; in
// the others the two are within 11 us of each other.  Measured (us per step, blocks
// against colours): Q2 64^3 FP32 333 / 366, FP64 568 / 471; Q2 32^3 87 / 163, 117 /
// 140; Q1 64^3 34 / 60, 51 / 66; Q1 128^3 170 / 186, 304 / 234; Q1 129 x 129 x 9 nodes
// FP32 86 / 39, 201 x 201 x 9 203 / 51, 65 x 65 x 257 79 / 109; N_Q1 48^3 (1334
// blocks) 64 / 39.
static void block_gain(const Level &L, int num_sms, const std::vector<int> &blk, const std::vector<unsigned> &ins,
                       const std::vector<int> &phase_of_row, const std::vector<std::vector<int>> &slices, int ncol,
                       double gain[2]) {
  constexpr double LAUNCH = 2.7, MB[2] = {0.4, 0.2}, SLICE[2] = {0.0184, 0.036}, CHUNK[2] = {0.0093, 0.016},
                   START = 3.6;
  const int P = (int)slices.size();
  std::vector<std::vector<double>> chunks(P);  // per pass
  for (int p = 0; p < P; p++) chunks[p].assign(slices[p].size(), 0.0);
  double inside = 0.0;
  for (int r = 0; r < L.Na; r++) {
    const int li = ins[r] & 0xffff, ui = ins[r] >> 16;
    chunks[phase_of_row[r]][blk[r]] += ((li + 3) / 4 + (ui + 3) / 4) / 64.0;
    inside += li + ui;
  }
  for (int t = 0; t < 2; t++) {
    double sweeps = 0.0;
    for (int p = 0; p < P; p++) {
      double most = 0.0, all = -START * num_sms;
      for (size_t b = 0; b < slices[p].size(); b++) {
        const double c = SLICE[t] * slices[p][b] + CHUNK[t] * chunks[p][b];
        most = std::max(most, c);
        all += c + START;
      }
      sweeps += 2.0 * std::max(most, all / num_sms);
    }
    gain[t] = LAUNCH * (2 * ncol - 2 - 4 * (P - 1)) + MB[t] * 1e-6 * inside * (t ? 10 : 6) - sweeps;
  }
}

// entries of each row in the solve copy: an active row keeps its columns < Na
// (columns are sorted, so that is a prefix), a Dirichlet row all of its own;
// nlow: those of lower colours, ins: those of lower / higher colours of the same
// phase (16 + 16 bits, saturated).  bad: two rows of one colour are coupled
// (BAD_COUPLED), a row is too long for the 16-bit source index (BAD_LONG).
enum { BAD_COUPLED = 1, BAD_LONG = 2 };
__global__ void k_row_counts(int N, int Na, const int *__restrict__ rp, const int *__restrict__ kc,
                             const int *__restrict__ colour, const int *__restrict__ phase, int *__restrict__ alen,
                             int *__restrict__ nlow, unsigned *__restrict__ ins, int *bad) {
  const int lane = threadIdx.x & 31;
  for (int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < N; r += (gridDim.x * blockDim.x) >> 5) {
    const int b = rp[r], e = rp[r + 1];
    int n = 0, low = 0, li = 0, ui = 0;
    bool same = false;
    if (r < Na) {
      const int cr = colour[r], pr = phase[cr];
      for (int k = b + lane; k < e; k += 32) {
        const int j = kc[k];
        if (j >= Na) break;
        n++;
        const int c = colour[j];
        low += c < cr;
        same |= c == cr && j != r;
        if (pr >= 0 && phase[c] == pr) {
          li += c < cr;
          ui += c > cr;
        }
      }
      n = __reduce_add_sync(0xffffffffu, n);
      low = __reduce_add_sync(0xffffffffu, low);
      li = __reduce_add_sync(0xffffffffu, li);
      ui = __reduce_add_sync(0xffffffffu, ui);
    } else {
      n = e - b;
    }
    same = __any_sync(0xffffffffu, same);
    if (lane == 0) {
      if (same) atomicOr(bad, BAD_COUPLED);
      if (n >= SELL_NO_SRC) atomicOr(bad, BAD_LONG);
      alen[r] = n;
      nlow[r] = low;
      ins[r] = (unsigned)min(li, 65535) | (unsigned)min(ui, 65535) << 16;
    }
  }
}

// The slices' columns, one warp per slice: 32-bit ones for every slice (the one-
// launch coarse cycle reads these), and column - row in 16 bits for the slices
// where every delta fits, which the sweeps and products read instead (2 bytes
// per entry, not 4); padding repeats the row (delta 0), padding lanes read x[0]
// with value 0.  src: position of the entry in its CSR row (SELL_NO_SRC:
// padding; without the split the diagonal step and the rest follow the row's
// own order instead, see k_csr_to_sell).  loc: the entries inside the block as
// slots of the block (padding: the row's own), in chunks of 4 steps,
// [chunk][lane][4], lower part, then higher.  nnz: entries stored in narrow and
// wide slices.
__global__ void k_sell_fill(int nslices, int Na, bool split, const int *__restrict__ perm, const int *__restrict__ sptr,
                            const int *__restrict__ nlow, const int *__restrict__ in, const int *__restrict__ lptr,
                            const int *__restrict__ rp, const int *__restrict__ kc, const int *__restrict__ alen,
                            const int *__restrict__ colour, const int *__restrict__ phase, const int *__restrict__ slot,
                            int *__restrict__ col, short *__restrict__ c16, unsigned short *__restrict__ src,
                            unsigned short *__restrict__ loc, unsigned char *__restrict__ wide,
                            unsigned long long *nnz) {
  const int lane = threadIdx.x & 31;
  for (int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < nslices; s += (gridDim.x * blockDim.x) >> 5) {
    const size_t off = (size_t)sptr[s] + lane;
    const int steps = (sptr[s + 1] - sptr[s]) / 32;
    const int r = perm[s * 32 + lane], low = nlow[s], low_in = in[s] & 0xffff, up_in = in[s] >> 16;
    const int ch_low = (low_in + 3) / 4, ch_up = (up_in + 3) / 4;
    const int len = r >= 0 ? alen[r] : 0, beg = r >= 0 ? rp[r] : 0;
    for (int j = 0; j < steps; j++) {
      col[off + 32 * (size_t)j] = r >= 0 ? r : 0;
      c16[off + 32 * (size_t)j] = 0;
      if (split) src[off + 32 * (size_t)j] = SELL_NO_SRC;
    }
    const bool active = r >= 0 && r < Na && split;
    const int cr = active ? colour[r] : 0, pr = active ? phase[cr] : -1;
    for (int j = 0; j < 4 * (ch_low + ch_up); j++)
      loc[((size_t)(lptr[s] + j / 4) * 32 + lane) * 4 + j % 4] = (unsigned short)(active ? slot[r] : 0);
    // next free step of each part: lower outside / inside the block, higher inside / outside
    int j_lo = 0, j_li = low - low_in, j_ui = low + 1, j_uo = low + 1 + up_in;
    bool fits = true;
    for (int k = 0; k < len; k++) {
      const int c = kc[beg + k];
      int j;
      if (c == r) {
        j = low;
      } else if (!active) {
        j = j_uo++;
      } else {
        const int cc = colour[c];
        const bool inside = pr >= 0 && phase[cc] == pr;
        j = cc < cr ? (inside ? j_li++ : j_lo++) : (inside ? j_ui++ : j_uo++);
        if (inside) {
          const int q = cc < cr ? j - (low - low_in) : 4 * ch_low + j - low - 1;
          loc[((size_t)(lptr[s] + q / 4) * 32 + lane) * 4 + q % 4] = (unsigned short)slot[c];
        }
      }
      const size_t p = off + 32 * (size_t)j;
      col[p] = c;
      const int d = c - r;
      if (d < -32768 || d > 32767) fits = false;
      c16[p] = (short)d;
      if (split) src[p] = (unsigned short)k;
    }
    const bool all = __all_sync(0xffffffffu, fits);
    const int stored = __reduce_add_sync(0xffffffffu, len);
    if (lane == 0) {
      wide[s] = all ? 0 : 1;
      atomicAdd(nnz + (all ? 0 : 1), (unsigned long long)stored);
    }
  }
}

int build_sell(Handle &h, Level &L) {
  if (L.sell_ready) return PMG_OK;
  const int N = L.N, Na = L.Na;
  const std::vector<int> &rp = L.h_rowptr, &kc = L.h_kcol;
  if ((int)rp.size() != N + 1) {
    set_error("build_sell: host copy of the CSR pattern missing");
    return PMG_ERR_STATE;
  }
  const int nc = (int)L.rcolor_ptr.size() - 1;
  std::vector<int> colour(N, nc);
  for (int g = 0; g < nc; g++)
    for (int k = L.rcolor_ptr[g]; k < L.rcolor_ptr[g + 1]; k++) colour[L.h_row_list[k]] = g;
  // device scratch of the set-up, in one allocation that stays with the handle
  // (an allocation can take longer than all the kernels here)
  // (a slice holds a row, so there are at most N; even parts keep 8-byte alignment)
  const size_t part = ((size_t)N + nc + 64) / 2 * 2;
  size_t most = part;  // (the largest level's at once, not level by level)
  for (const Level &o : h.lv) most = std::max(most, ((size_t)o.N + o.rcolor_ptr.size() + 64) / 2 * 2);
  PMG_TRY(h.setup_scratch.reserve(8 * most));
  int *d_colour = h.setup_scratch.p, *d_phase = d_colour + part, *d_nlow = d_phase + part, *d_lptr = d_nlow + part,
      *d_slot = d_lptr + part, *d_rowa = d_slot + part, *d_alen = d_rowa + part, *d_bad = d_alen + part;
  std::vector<int> blk;  // block of each active row inside its phase
  std::vector<std::vector<int>> blk_slices;
  auto put = [&](int *d, const std::vector<int> &v) {
    return v.empty() ? cudaSuccess
                     : cudaMemcpyAsync(d, v.data(), sizeof(int) * v.size(), cudaMemcpyHostToDevice, h.stream);
  };
  PMG_CUDA(put(d_colour, colour));
  PMG_TRY(find_blocks(h, L, colour, blk, blk_slices, d_colour, d_phase, d_nlow, d_rowa));
  std::vector<int> phase(nc + 1, -1);
  for (size_t p = 0; p + 1 < L.blk_col.size(); p++)
    for (int c = L.blk_col[p]; c < L.blk_col[p + 1]; c++) phase[c] = (int)p;
  // the rows' counts (k_row_counts).  A pattern that couples two rows of one
  // colour (possible for an unsymmetric one), or has a row too long for the
  // 16-bit source index, is not split: every off-diagonal entry counts as of a
  // higher colour and the sweeps read whole rows.
  std::vector<int> alen(N), nlow(N);
  std::vector<unsigned> ins(N);
  unsigned *d_ins = reinterpret_cast<unsigned *>(d_rowa);
  int bad = 0;
  PMG_CUDA(put(d_phase, phase));
  PMG_CUDA(cudaMemsetAsync(d_bad, 0, 8 * sizeof(int), h.stream));
  k_row_counts<<<h.num_sms * 8, 256, 0, h.stream>>>(N, Na, L.rowptr.p, L.kcol.p, d_colour, d_phase, d_alen, d_nlow,
                                                    d_ins, d_bad);
  count_launches(1);
  PMG_CUDA(cudaGetLastError());
  PMG_CUDA(cudaMemcpyAsync(alen.data(), d_alen, sizeof(int) * N, cudaMemcpyDeviceToHost, h.stream));
  PMG_CUDA(cudaMemcpyAsync(nlow.data(), d_nlow, sizeof(int) * N, cudaMemcpyDeviceToHost, h.stream));
  PMG_CUDA(cudaMemcpyAsync(ins.data(), d_ins, sizeof(int) * N, cudaMemcpyDeviceToHost, h.stream));
  PMG_CUDA(cudaMemcpyAsync(&bad, d_bad, sizeof(int), cudaMemcpyDeviceToHost, h.stream));
  PMG_CUDA(cudaStreamSynchronize(h.stream));
  bool split = bad == 0;
  L.blk_on[0] = L.blk_on[1] = false;
  if (!L.blk_col.empty()) {
    std::vector<int> phase_of_row(Na);
    bool fits = split;  // (the blocks' tables keep the inside counts in 12 bits)
    for (int r = 0; r < Na; r++) {
      phase_of_row[r] = phase[colour[r]];
      fits = fits && (ins[r] & 0xffff) <= 4095 && ins[r] >> 16 <= 4095;
    }
    double gain[2];
    block_gain(L, h.num_sms, blk, ins, phase_of_row, blk_slices, nc, gain);
    size_t largest = 0;
    for (const auto &p : blk_slices)
      for (int s : p) largest = std::max(largest, (size_t)s);
    for (int t = 0; t < 2; t++)
      L.blk_on[t] = fits && gain[t] > 0.0 && largest * ((t ? 8 : 4) * 32 + BLK_TASK) <= BLK_SMEM;
    // rows sorted by blocks are scattered and padded, which costs colour launches: the
    // level is laid out for blocks only if the precision in use sweeps by them (Q2
    // 64^3 FP64 V-cycle, finest level by colours: 3.52 ms with the rows by blocks, 3.12
    // without; by blocks 3.56)
    if (!L.blk_on[h.prm.precision == PMG_PREC_FP64]) {
      L.blk_on[0] = L.blk_on[1] = false;
      L.blk_col.clear();
      std::fill(phase.begin(), phase.end(), -1);
      std::fill(ins.begin(), ins.end(), 0u);
    }
  }
  std::vector<int> dd_row, dd_beg;
  for (int r = 0; r < Na; r++)
    if (rp[r] + alen[r] < rp[r + 1]) {
      dd_row.push_back(r);
      dd_beg.push_back(rp[r] + alen[r]);
    }
  std::vector<int> perm, group_slice, sptr, snlow, sin, lptr;
  long total, total_in;
  int nslices;
  for (;;) {
    if (!split) {
      std::fill(nlow.begin(), nlow.end(), 0);
      std::fill(ins.begin(), ins.end(), 0u);
      L.blk_col.clear();
      L.blk_on[0] = L.blk_on[1] = false;
    }
    const bool blocks = !L.blk_col.empty();
    // groups: colours of the active rows (block by block), then the Dirichlet rows
    std::vector<std::vector<int>> group(nc + 1);
#pragma omp parallel for schedule(dynamic, 1)
    for (int g = 0; g <= nc; g++) {
      std::vector<int> rows, &out = group[g];
      if (g < nc) rows.assign(L.h_row_list.begin() + L.rcolor_ptr[g], L.h_row_list.begin() + L.rcolor_ptr[g + 1]);
      else for (int r = Na; r < N; r++) rows.push_back(r);
      const bool by_block = blocks && g < nc;
      // by block, then longest row, longest lower part, most inside entries first (the
      // keys side by side: a comparator that looks them up takes three times as long)
      struct Key {
        int blk, len, low;
        unsigned ins;
        int row;
      };
      std::vector<Key> key(rows.size());
      for (size_t k = 0; k < rows.size(); k++) {
        const int r = rows[k];
        key[k] = {by_block ? blk[r] : 0, alen[r], nlow[r], r < Na ? ins[r] : 0u, r};
      }
      std::sort(key.begin(), key.end(), [](const Key &a, const Key &b) {
        if (a.blk != b.blk) return a.blk < b.blk;
        if (a.len != b.len) return a.len > b.len;
        if (a.low != b.low) return a.low > b.low;
        if (a.ins != b.ins) return a.ins > b.ins;
        return a.row < b.row;
      });
      out.reserve(rows.size() + 32);
      for (size_t k = 0; k < key.size(); k++) {
        if (k > 0 && key[k].blk != key[k - 1].blk)
          while (out.size() % 32) out.push_back(-1);
        out.push_back(key[k].row);
      }
      while (out.size() % 32) out.push_back(-1);
    }
    perm.clear();
    perm.reserve((size_t)N + 32 * (nc + 1));
    group_slice.assign(nc + 2, 0);
    for (int g = 0; g <= nc; g++) {
      group_slice[g] = (int)(perm.size() / 32);
      perm.insert(perm.end(), group[g].begin(), group[g].end());
    }
    group_slice[nc + 1] = nslices = (int)(perm.size() / 32);
    sptr.assign(nslices + 1, 0);
    snlow.assign(nslices, 0);
    sin.assign(nslices, 0);
    lptr.assign(nslices + 1, 0);
    total = total_in = 0;
    for (int s = 0; s < nslices && total <= 2147483647L; s++) {
      int low_out = 0, low_in = 0, up_in = 0, up_out = 0;
      for (int l = 0; l < 32; l++) {
        const int r = perm[(size_t)s * 32 + l];
        if (r < 0) continue;
        const int li = ins[r] & 0xffff, ui = ins[r] >> 16;
        low_out = std::max(low_out, nlow[r] - li);
        low_in = std::max(low_in, li);
        up_in = std::max(up_in, ui);
        up_out = std::max(up_out, alen[r] - 1 - nlow[r] - ui);
      }
      sptr[s] = (int)total;
      lptr[s] = (int)total_in;
      snlow[s] = low_out + low_in;
      sin[s] = low_in | up_in << 16;
      total += 32L * (low_out + low_in + 1 + up_in + up_out);
      total_in += (low_in + 3) / 4 + (up_in + 3) / 4;  // chunks of 4 steps
    }
    if (total <= 2147483647L) break;
    if (!split) {
      set_error("build_sell: padded matrix exceeds 2^31 entries");
      return PMG_ERR_UNSUPPORTED;
    }
    split = false;  // whole rows pad less
  }
  sptr[nslices] = (int)total;
  lptr[nslices] = (int)total_in;
  // slots of the rows in their blocks, and the blocks' slices in hop order
  const bool blocks = !L.blk_col.empty();
  std::vector<int> slot, tab, meta, brows;
  L.blk_tab0.clear();
  L.blk_slots.clear();
  if (blocks) {
    slot.assign(Na, 0);
    for (size_t p = 0; p + 1 < L.blk_col.size(); p++) {
      const int c0 = L.blk_col[p], w = L.blk_col[p + 1] - c0, nb = L.blk_n[p];
      // slices of every block and colour
      std::vector<int> beg((size_t)nb * w, 0), cnt((size_t)nb * w, 0);
      for (int c = 0; c < w; c++)
        for (int s = group_slice[c0 + c]; s < group_slice[c0 + c + 1]; s++) {
          const size_t k = (size_t)blk[perm[(size_t)s * 32]] * w + c;
          if (cnt[k]++ == 0) beg[k] = s;
        }
      const size_t t0 = tab.size();
      L.blk_tab0.push_back((int)t0);
      tab.resize(t0 + (size_t)nb * (w + 2));
      int slots = 0;
      for (int b = 0; b < nb; b++) {
        int *t = &tab[t0 + (size_t)b * (w + 2)], ord = 0;
        t[0] = (int)(meta.size() / 4);
        for (int c = 0; c < w; c++) {
          t[1 + c] = ord;
          for (int s = beg[(size_t)b * w + c], e = s + cnt[(size_t)b * w + c]; s < e; s++, ord++) {
            const int li = sin[s] & 0xffff, ui = sin[s] >> 16;
            meta.insert(meta.end(), {lptr[s], li | ui << 12 | c << 24, s, 0});
            for (int l = 0; l < 32; l++) {
              const int r = perm[(size_t)s * 32 + l];
              brows.push_back(r);
              if (r >= 0) slot[r] = ord * 32 + l;
            }
          }
        }
        t[1 + w] = ord;
        slots = std::max(slots, ord * 32);
      }
      L.blk_slots.push_back(slots);
    }
  }
  // one allocation; its first part comes from the host in one copy
  L.n_dd = (int)dd_row.size();
  Carve parts;
  parts.add(L.sell_perm, perm.size());
  parts.add(L.sell_ptr, sptr.size());
  parts.add(L.sell_nlow, snlow.size());
  parts.add(L.sell_in, sin.size());
  parts.add(L.blk_tab, tab.size());
  parts.add(L.blk_meta, meta.size());
  parts.add(L.blk_rows, brows.size());
  parts.add(L.dd_row, dd_row.size());
  parts.add(L.dd_beg, dd_beg.size());
  std::vector<unsigned char> host(parts.bytes);
  {
    const std::vector<int> *from[] = {&perm, &sptr, &snlow, &sin, &tab, &meta, &brows, &dd_row, &dd_beg};
    for (size_t k = 0; k < parts.parts.size(); k++)
      if (!from[k]->empty()) memcpy(&host[parts.parts[k].second], from[k]->data(), from[k]->size() * sizeof(int));
  }
  parts.add(L.sell_alen, N);
  parts.add(L.sell_wide, nslices);
  parts.add(L.sell_col, total);
  parts.add(L.sell_c16, total);
  parts.add(L.sell_src, split ? total : 0);
  parts.add(L.sell_loc, (size_t)total_in * 128);
  PMG_TRY(parts.place(L.sell_mem));
  if (!host.empty())
    PMG_CUDA(cudaMemcpyAsync(L.sell_mem.p, host.data(), host.size(), cudaMemcpyHostToDevice, h.stream));
  PMG_CUDA(cudaMemcpyAsync(L.sell_alen.p, d_alen, sizeof(int) * N, cudaMemcpyDeviceToDevice, h.stream));
  // the slices' columns, filled on the device
  unsigned long long *d_nnz = reinterpret_cast<unsigned long long *>(d_bad + 2), nnz[2] = {0, 0};
  PMG_CUDA(put(d_lptr, lptr));
  PMG_CUDA(put(d_slot, slot));
  PMG_CUDA(put(d_phase, phase));
  if (nslices > 0) {
    k_sell_fill<<<std::min((nslices + 7) / 8, h.num_sms * 16), 256, 0, h.stream>>>(
        nslices, Na, split, L.sell_perm.p, L.sell_ptr.p, L.sell_nlow.p, L.sell_in.p, d_lptr, L.rowptr.p, L.kcol.p,
        L.sell_alen.p, d_colour, d_phase, d_slot, L.sell_col.p, L.sell_c16.p, L.sell_src.p, L.sell_loc.p,
        L.sell_wide.p, d_nnz);
    count_launches(1);
    PMG_CUDA(cudaGetLastError());
  }
  PMG_CUDA(cudaMemcpyAsync(nnz, d_nnz, sizeof(nnz), cudaMemcpyDeviceToHost, h.stream));
  PMG_CUDA(cudaStreamSynchronize(h.stream));
  // these belong to the old layout
  L.sums_mem32.release();
  L.sums_mem64.release();
  L.blk_mem32.release();
  L.blk_mem64.release();
  L.blk_chunks = total_in;
  L.sell_group = group_slice;
  L.sell_nslices = nslices;
  L.sell_nnz = total;
  L.sell_split = split;
  L.sell_coupled = (bad & BAD_COUPLED) != 0;
  L.sell_nnz_narrow = (long)nnz[0];
  L.sell_nnz_wide = (long)nnz[1];
  L.sell_ready = true;
  L.sell_val_fresh32 = L.sell_val_fresh64 = false;
  return PMG_OK;
}

// values of the CSR matrix into the slice layout (and the permuted inverse
// diagonal): through the source index, or, for a pattern that is not split,
// the diagonal first and the row's other entries in their order
template <typename T>
__global__ void k_csr_to_sell(int nslices, const int *__restrict__ perm, const int *__restrict__ sptr,
                              const int *__restrict__ rp, const int *__restrict__ alen, const double *__restrict__ a,
                              const int *__restrict__ dpos, const unsigned short *__restrict__ src,
                              T *__restrict__ val, T *__restrict__ invd) {
  const int lane = threadIdx.x & 31;
  for (int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < nslices; s += (gridDim.x * blockDim.x) >> 5) {
    const int off = sptr[s], steps = (sptr[s + 1] - off) >> 5;
    const int r = perm[s * 32 + lane];
    const int beg = r >= 0 ? rp[r] : 0, len = r >= 0 ? alen[r] : 0;
    const int dp = r >= 0 ? dpos[r] - beg : 0;
    if (src) {
#pragma unroll 8
      for (int j = 0; j < steps; j++) {
        const int q = __ldcs(src + off + 32 * j + lane);
        val[off + 32 * j + lane] = q != SELL_NO_SRC ? (T)a[beg + q] : (T)0;
      }
    } else {
      for (int j = 0; j < steps; j++) {
        const int q = j == 0 ? dp : j - 1 + (j - 1 >= dp);
        val[off + 32 * j + lane] = q < len ? (T)a[beg + q] : (T)0;
      }
    }
    T dv = (T)1;
    if (r >= 0) {
      const double d = a[beg + dp];
      dv = (T)(d != 0.0 ? 1.0 / d : 1.0);
    }
    invd[s * 32 + lane] = dv;
  }
}

// the sums kept between the sweeps, zero at first (the first colour's lower and
// the last colour's upper sums stay 0, the Dirichlet rows' too)
template <typename T>
static int alloc_sums(Handle &h, const Level &L, DBuf<unsigned char> &mem, View<T> &sl, View<T> &su) {
  if (mem.p) return PMG_OK;  // (released with the layout)
  const size_t n = (size_t)L.sell_nslices * 32;
  Carve parts;
  parts.add(sl, n);
  parts.add(su, n);
  PMG_TRY(parts.place(mem));
  PMG_CUDA(cudaMemsetAsync(mem.p, 0, mem.n, h.stream));
  return PMG_OK;
}

// the entries inside the blocks a second time, in the block kernel's layout
// ([chunk of 4 steps][lane][4]: one 16-byte load per lane and chunk in FP32)
template <typename T>
__global__ void k_blk_values(int n, const int4 *__restrict__ meta, const int *__restrict__ sptr,
                             const int *__restrict__ nlow, const T *__restrict__ val, T *__restrict__ bval) {
  const int lane = threadIdx.x & 31;
  for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += (gridDim.x * blockDim.x) >> 5) {
    const int4 m = __ldg(meta + i);
    const int li = m.y & 0xfff, ui = m.y >> 12 & 0xfff, s = m.z, low = __ldg(nlow + s);
    const size_t off = (size_t)__ldg(sptr + s) + lane;
    T *out = bval + (size_t)m.x * 128 + lane * 4;
    for (int j = 0; j < (li + 3) / 4 * 4; j++)
      out[j / 4 * 128 + j % 4] = j < li ? val[off + 32 * (size_t)(low - li + j)] : (T)0;
    out += (li + 3) / 4 * 128;
    for (int j = 0; j < (ui + 3) / 4 * 4; j++)
      out[j / 4 * 128 + j % 4] = j < ui ? val[off + 32 * (size_t)(low + 1 + j)] : (T)0;
  }
}

template <typename T>
int sell_values(Handle &h, Level &L) {
  const bool f32 = sizeof(T) == 4;
  if (f32 ? L.sell_val_fresh32 : L.sell_val_fresh64) return PMG_OK;
  PMG_TRY(build_sell(h, L));
  T *val, *invd;
  if (f32) {
    Carve parts;
    parts.add(L.sell_val32, L.sell_nnz);
    parts.add(L.sell_invd32, (size_t)L.sell_nslices * 32);
    PMG_TRY(parts.place(L.val_mem32));
    val = reinterpret_cast<T *>(L.sell_val32.p);
    invd = reinterpret_cast<T *>(L.sell_invd32.p);
  } else {
    Carve parts;
    parts.add(L.sell_val64, L.sell_nnz);
    parts.add(L.sell_invd64, (size_t)L.sell_nslices * 32);
    PMG_TRY(parts.place(L.val_mem64));
    val = reinterpret_cast<T *>(L.sell_val64.p);
    invd = reinterpret_cast<T *>(L.sell_invd64.p);
  }
  int blocks = std::min((L.sell_nslices + 7) / 8, h.num_sms * 16);
  k_csr_to_sell<T><<<std::max(blocks, 1), 256, 0, h.stream>>>(L.sell_nslices, L.sell_perm.p, L.sell_ptr.p, L.rowptr.p,
                                                                L.sell_alen.p, L.A.p, L.diagpos.p,
                                                                L.sell_split ? L.sell_src.p : nullptr, val, invd);
  count_launches(1);
  PMG_CUDA(cudaGetLastError());
  if (f32) L.sell_val_fresh32 = true, L.blk_val_fresh32 = false;
  else L.sell_val_fresh64 = true, L.blk_val_fresh64 = false;
  return PMG_OK;
}
template int sell_values<float>(Handle &, Level &);
template int sell_values<double>(Handle &, Level &);

// A block of K warps owns one slice: warp w accumulates the column steps
// j = w, w+K, ... of the slice's 32 rows (coalesced 32-wide loads), the K
// partial sums meet in shared memory and warp 0 finishes the rows.  K is
// chosen per launch (4, 8 or 16): small colours get more warps per slice so
// that each warp's chain of dependent loads (column index, then x) stays
// short; large colours already fill the GPU with K = 4.

// Column indices: a slice whose deltas fit (every slice of a lattice-ordered
// level) is read as 16-bit column - row deltas and gathered through x + row
// of the lane; the other slices read the 32-bit columns.  The choice is per
// slice and warp-uniform.  Matrix values and columns are read once per pass
// with streaming loads (ld.global.cs, evict-first), so they do not push the
// gathered iterate out of L1/L2: measured on the 64^3 finest level, FP32 SSOR
// step 0.490 -> 0.467 ms, FP64 SpMV 0.296 -> 0.272 ms.
template <int PF, int K>
__device__ __forceinline__ void sell_load_cols(bool wd, const int *__restrict__ col, const short *__restrict__ c16,
                                               int base, int j0, int lmax, int *ci) {
  if (wd) {
#pragma unroll
    for (int u = 0; u < PF; u++) ci[u] = j0 + u * K < lmax ? __ldcs(col + base + 32 * K * u) : 0;
  } else {
#pragma unroll
    for (int u = 0; u < PF; u++) ci[u] = j0 + u * K < lmax ? (int)__ldcs(c16 + base + 32 * K * u) : 0;
  }
}

// y = A x (MODE 0), d = f - A x (MODE 1), the Jacobi update
// y = x + omega (f - A x) / a_rr (MODE 2, into a vector other than x), or the
// defect after an SSOR step (MODE 3): the step's backward sweep has left the
// sums over the higher colours of the final x in su, so only the lower part
// and the diagonal are read.  The Dirichlet rows (slices from sd on) have no
// colours and are read whole: a caller's matrix may hold more than the diagonal
// there, and a transfer may take their defect to active rows.  Over slices [s0, s1)
template <typename T, int MODE, int K>
__global__ void __launch_bounds__(32 * K) k_sell_mv(int s0, int s1, int sd, const int *__restrict__ perm,
                                                    const int *__restrict__ sptr, const int *__restrict__ nlow,
                                                    const int *__restrict__ col, const short *__restrict__ c16,
                                                    const unsigned char *__restrict__ wide,
                                                    const T *__restrict__ val, const T *__restrict__ x,
                                                    const T *__restrict__ f, T *__restrict__ y,
                                                    const T *__restrict__ invd, const T *__restrict__ su, T omega) {
  // column steps per chunk: measured on the 64^3 Q2 finest level, FP64
  // product 0.275 ms with 8, 0.252 with 4, 0.253 with 2; FP32 defect 0.186
  // ms with 16, 0.164 with 8, 0.173 with 4
  constexpr int PF = sizeof(T) == 4 ? 8 : 4;
  __shared__ T part[K][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int s = s0 + blockIdx.x;
  int off = 0, lmax = 0, r = -1;
  bool wd = false;
  int ci[PF];
  T cv[PF];
  auto load_chunk = [&](int c0) {
    const int j0 = w + c0 * K;
    sell_load_cols<PF, K>(wd, col, c16, off + 32 * j0 + lane, j0, lmax, ci);
#pragma unroll
    for (int u = 0; u < PF; u++) cv[u] = j0 + u * K < lmax ? __ldcs(val + off + 32 * (j0 + u * K) + lane) : (T)0;
  };
  auto start = [&](int sl) {
    off = __ldg(sptr + sl);
    lmax = MODE == 3 && sl < sd ? __ldg(nlow + sl) + 1 : (__ldg(sptr + sl + 1) - off) >> 5;
    wd = __ldg(wide + sl) != 0;
    r = __ldg(perm + sl * 32 + lane);
    load_chunk(0);
  };
  // the matrix is not written by the predecessor: its first chunk streams in while that drains
  if (s < s1) start(s);
  pdl_wait();
  pdl_trigger();
  for (; s < s1; s += gridDim.x) {
    const T *xb = wd ? x : x + (r > 0 ? r : 0);
    T sum = 0;
    for (int c0 = 0;; c0 += PF) {
#pragma unroll
      for (int u = 0; u < PF; u++)
        if (w + (c0 + u) * K < lmax) sum += cv[u] * __ldg(xb + ci[u]);
      if (w + (c0 + PF) * K >= lmax) break;
      load_chunk(c0 + PF);
    }
    part[w][lane] = sum;
    const int rr = r;
    const int sn = s + gridDim.x;
    if (sn < s1) start(sn);  // next slice's first chunk before the reduction
    __syncthreads();
    if (w == 0) {
#pragma unroll
      for (int k = 1; k < K; k++) sum += part[k][lane];
      if (rr >= 0) {
        if (MODE == 3) y[rr] = __ldg(f + rr) - (sum + __ldg(su + s * 32 + lane));
        else if (MODE == 2) y[rr] = __ldg(x + rr) + omega * (__ldg(f + rr) - sum) * __ldg(invd + s * 32 + lane);
        else y[rr] = MODE ? __ldg(f + rr) - sum : sum;
      }
    }
    __syncthreads();
  }
}

// Gauss-Seidel update of the rows of one colour (slices [s0, s1)):
//   x_r := (1 - omega) x_r + omega (f_r - lower - upper) / a_rr
// with lower / upper the sums over the columns of lower / higher colours.
// A sweep reads one side of the diagonal only: when the forward sweep reaches
// colour c, the columns of higher colours still hold what the previous backward
// sweep left, and their sum was formed there; in the backward sweep the same
// goes for the lower colours.  So a forward pass (GS_LOWER) reads the lower
// part, takes `upper` from su and leaves `lower` in sl; a backward pass
// (GS_UPPER) reads the upper part, takes `lower` from sl and leaves `upper` in
// su (both in the slices' order).  Every entry is read once per SSOR step
// instead of twice.  The sums are the same ones, so the iterate differs by
// rounding only.  GS_LOWER_ZERO: the first sweep from x = 0, where `upper` is
// 0.  GS_FULL: the first forward sweep over an arbitrary x (after the
// prolongation), and every SOR sweep, forms both sums.
// The first chunk of column steps of a warp's slice is loaded before
// pdl_wait(): the predecessor in the stream (the previous colour, a transfer
// or a defect) writes vectors only, never the matrix, so the colour's matrix
// streams in while the predecessor drains, and only the x gathers wait.
enum { GS_LOWER = 0, GS_LOWER_ZERO = 1, GS_UPPER = 2, GS_FULL = 3 };

template <typename T, int K, int MODE>
__global__ void __launch_bounds__(32 * K) k_sell_gs(int s0, int s1, const int *__restrict__ perm,
                                                    const int *__restrict__ sptr, const int *__restrict__ nlow,
                                                    const int *__restrict__ col, const short *__restrict__ c16,
                                                    const unsigned char *__restrict__ wide,
                                                    const T *__restrict__ val, const T *__restrict__ invd,
                                                    const T *__restrict__ f, T *x, T *sl, T *su, T omega) {
  constexpr bool FULL = MODE == GS_FULL;
  constexpr int GS_PF = FULL ? (sizeof(T) == 4 ? 16 : 8) : (sizeof(T) == 4 ? 8 : 8);  // column steps per chunk
  __shared__ T part[K][32], part_up[FULL ? K : 1][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int s = s0 + blockIdx.x;
  int off = 0, n = 0, nl = 0, r = -1;  // n column steps from off; nl: the lower ones among all (FULL)
  bool wd = false;
  T id = 0;
  int ci[GS_PF];
  T cv[GS_PF];
  auto load_chunk = [&](int c0) {
    const int j0 = w + c0 * K;
    sell_load_cols<GS_PF, K>(wd, col, c16, off + 32 * j0 + lane, j0, n, ci);
#pragma unroll
    for (int u = 0; u < GS_PF; u++)
      cv[u] = j0 + u * K < n ? __ldcs(val + off + 32 * (j0 + u * K) + lane) : (T)0;
  };
  auto prefetch = [&](int q) {
    off = __ldg(sptr + q);
    n = (__ldg(sptr + q + 1) - off) >> 5;
    nl = __ldg(nlow + q);
    if (MODE == GS_UPPER) {
      off += 32 * (nl + 1);
      n -= nl + 1;
    } else if (!FULL) {
      n = nl;
    }
    wd = __ldg(wide + q) != 0;
    r = __ldg(perm + q * 32 + lane);
    if (w == 0) id = __ldg(invd + q * 32 + lane);
    load_chunk(0);
  };
  if (s < s1) prefetch(s);
  pdl_wait();
  pdl_trigger();
  for (; s < s1; s += gridDim.x) {
    const T *xb = wd ? x : x + (r > 0 ? r : 0);
    T rest = 0, xr = 0;  // f minus the sum that is not formed here; the old value (omega != 1)
    if (w == 0 && r >= 0) {
      rest = __ldg(f + r);
      if (MODE == GS_LOWER) rest -= su[s * 32 + lane];
      if (MODE == GS_UPPER) rest -= sl[s * 32 + lane];
      if (omega != (T)1) xr = x[r];
    }
    T sum = 0, up = 0;
    // column steps in chunks of GS_PF: the gathers of a chunk go out, then the
    // next chunk's column / value loads, so a long row costs one latency per chunk
    for (int c0 = 0;; c0 += GS_PF) {
#pragma unroll
      for (int u = 0; u < GS_PF; u++) {
        const int j = w + (c0 + u) * K;
        if (j < n) {
          const T t = cv[u] * xb[ci[u]];
          if (!FULL || j < nl) sum += t;
          else if (j > nl) up += t;
        }
      }
      if (w + (c0 + GS_PF) * K >= n) break;
      load_chunk(c0 + GS_PF);
    }
    part[w][lane] = sum;
    if (FULL) part_up[FULL ? w : 0][lane] = up;
    __syncthreads();
    if (w == 0) {
#pragma unroll
      for (int k = 1; k < K; k++) {
        sum += part[k][lane];
        if (FULL) up += part_up[FULL ? k : 0][lane];
      }
      if (r >= 0) {
        const T v = (FULL ? rest - (sum + up) : rest - sum) * id;
        x[r] = omega != (T)1 ? xr + omega * (v - xr) : v;
        if (MODE == GS_UPPER) su[s * 32 + lane] = sum;
        else sl[s * 32 + lane] = sum;
      }
    }
    __syncthreads();
    if (s + gridDim.x < s1) prefetch(s + gridDim.x);
  }
}

// warps per slice for a launch over `slices` slices: the smallest K (>= 4;
// K = 2 and deeper unrolling measured slower on the 64^3 finest level) that
// still gives every SM 32 warps, at most kmax
static int pick_k(int slices, int num_sms, int kmax = 16) {
  static int kmin = -1;
  if (kmin < 0) {
    const char *e = getenv("PMG_SELL_KMIN");
    kmin = e ? atoi(e) : 4;
    if (kmin != 2 && kmin != 8 && kmin != 16) kmin = 4;
  }
  const long want = 32L * num_sms;  // warps to keep the load pipes busy
  int k = kmin;
  while (k < kmax && (long)slices * k < want) k *= 2;
  return k;
}

// y_r -= sum over the Dirichlet columns j of active row r of A_rj v_j (the
// entries [dd_beg, row end) of the CSR row, FP64 values)
template <typename T>
__global__ void k_dirichlet_cols(int n, const int *__restrict__ rows, const int *__restrict__ beg,
                                 const int *__restrict__ rp, const int *__restrict__ kc, const double *__restrict__ a,
                                 const T *v, T *y, double sign) {
  pdl_wait();
  pdl_trigger();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int r = __ldg(rows + i);
  double s = 0;
  for (int k = __ldg(beg + i), e = __ldg(rp + r + 1); k < e; k++) s += __ldg(a + k) * (double)v[__ldg(kc + k)];
  y[r] = (T)((double)y[r] + sign * s);
}

template <typename T>
int dirichlet_cols(cudaStream_t s, const Level &L, const T *v, T *y, bool add) {
  if (L.n_dd == 0) return PMG_OK;
  PMG_CUDA(launch_pdl(k_dirichlet_cols<T>, dim3((L.n_dd + 255) / 256), dim3(256), 0, s, L.n_dd,
                      (const int *)L.dd_row.p, (const int *)L.dd_beg.p, (const int *)L.rowptr.p,
                      (const int *)L.kcol.p, (const double *)L.A.p, v, y, add ? 1.0 : -1.0));
  count_launches(1);
  return PMG_OK;
}
template int dirichlet_cols<float>(cudaStream_t, const Level &, const float *, float *, bool);
template int dirichlet_cols<double>(cudaStream_t, const Level &, const double *, double *, bool);

// grid of a SELL launch: one CTA per slice up to a cap, beyond which CTAs loop
// over slices (loading the next slice's first chunk before the reduction).
// Measured on the 64^3 Q2 finest level (K = 4, 4 / 8 column steps per chunk):
// 256 CTAs per SM, FP64 product 0.247 ms (64: 0.268, 1024: 0.252, the earlier
// 512: 0.252), FP32 defect 0.162 ms (64: 0.173, 128: 0.164, 1024: 0.165); a
// colour sweep stays below the cap.  PMG_SELL_CTAS_PER_SM overrides the cap.
template <typename T>
static int slice_grid(int nslices, int num_sms, int k) {
  static int cps = -1;
  if (cps < 0) {
    const char *e = getenv("PMG_SELL_CTAS_PER_SM");
    cps = e ? std::max(0, atoi(e)) : 0;
  }
  const long cap = (long)num_sms * (cps ? cps : 256);
  return (int)std::max(1L, std::min((long)nslices, cap));
}

template <typename T>
static const T *sell_val(const Level &L) {
  if (sizeof(T) == 4) return reinterpret_cast<const T *>(L.sell_val32.p);
  return reinterpret_cast<const T *>(L.sell_val64.p);
}
template <typename T>
static T *sell_sum(const Level &L, bool up) {
  if (sizeof(T) == 4) return reinterpret_cast<T *>(up ? L.sell_su32.p : L.sell_sl32.p);
  return reinterpret_cast<T *>(up ? L.sell_su64.p : L.sell_sl64.p);
}
template <typename T>
static const T *sell_invd(const Level &L) {
  if (sizeof(T) == 4) return reinterpret_cast<const T *>(L.sell_invd32.p);
  return reinterpret_cast<const T *>(L.sell_invd64.p);
}

template <typename T, int MODE, int K>
static cudaError_t launch_mv(cudaStream_t s, const Level &L, const T *x, const T *f, T *y, int num_sms, int n = -1,
                             T omega = 0) {
  if (n < 0) n = L.sell_nslices;
  return launch_pdl(k_sell_mv<T, MODE, K>, dim3(slice_grid<T>(n, num_sms, K)), dim3(32 * K), 0, s, 0, n,
                    L.sell_group[L.sell_group.size() - 2], (const int *)L.sell_perm.p, (const int *)L.sell_ptr.p, (const int *)L.sell_nlow.p,
                    (const int *)L.sell_col.p, (const short *)L.sell_c16.p, (const unsigned char *)L.sell_wide.p,
                    sell_val<T>(L), x, f, y, sell_invd<T>(L), (const T *)sell_sum<T>(L, true), omega);
}

template <typename T>
int sell_spmv(cudaStream_t s, const Level &L, const T *x, const T *f, T *y, int mode, int num_sms) {
  int k = pick_k(L.sell_nslices, num_sms);
  cudaError_t e;
  if (k < 4) k = 4;  // a full-matrix product has enough slices for K = 4
  if (mode == 3) e = k == 16 ? launch_mv<T, 3, 16>(s, L, x, f, y, num_sms) : k == 8 ? launch_mv<T, 3, 8>(s, L, x, f, y, num_sms)
                                                                                  : launch_mv<T, 3, 4>(s, L, x, f, y, num_sms);
  else if (mode) e = k == 16 ? launch_mv<T, 1, 16>(s, L, x, f, y, num_sms) : k == 8 ? launch_mv<T, 1, 8>(s, L, x, f, y, num_sms)
                                                                             : launch_mv<T, 1, 4>(s, L, x, f, y, num_sms);
  else e = k == 16 ? launch_mv<T, 0, 16>(s, L, x, f, y, num_sms) : k == 8 ? launch_mv<T, 0, 8>(s, L, x, f, y, num_sms)
                                                                          : launch_mv<T, 0, 4>(s, L, x, f, y, num_sms);
  PMG_CUDA(e);
  count_launches(1);
  return PMG_OK;
}
template int sell_spmv<float>(cudaStream_t, const Level &, const float *, const float *, float *, int, int);
template int sell_spmv<double>(cudaStream_t, const Level &, const double *, const double *, double *, int, int);

template <typename T>
__global__ void k_copy_active(int Na, const T *__restrict__ src, T *__restrict__ dst) {
  pdl_wait();
  pdl_trigger();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < Na) dst[i] = src[i];
}

// One damped Jacobi step (TMGLevel3D::Jacobi, MGLevel3D.C:469-560):
// x_a := x_a + omega (f_a - A_a x) / a_aa from the previous
// iterate, written into `tmp` (the active rows' slices are the colour groups)
// and copied back.  x_D = f_D already holds when a level's smoothing starts, so
// the previous Dirichlet values the reference keeps in its aux copy equal the
// new ones.
template <typename T>
int sell_jacobi(cudaStream_t s, const Level &L, const T *f, T *x, T *tmp, double omega, int num_sms) {
  const int nc = (int)L.sell_group.size() - 2;
  const int na_slices = L.sell_group[nc];
  if (na_slices <= 0) return PMG_OK;
  const int k = std::max(4, pick_k(na_slices, num_sms));
  cudaError_t e = k == 16 ? launch_mv<T, 2, 16>(s, L, x, f, tmp, num_sms, na_slices, (T)omega)
                : k == 8  ? launch_mv<T, 2, 8>(s, L, x, f, tmp, num_sms, na_slices, (T)omega)
                          : launch_mv<T, 2, 4>(s, L, x, f, tmp, num_sms, na_slices, (T)omega);
  PMG_CUDA(e);
  PMG_CUDA(launch_pdl(k_copy_active<T>, dim3((L.Na + 255) / 256), dim3(256), 0, s, L.Na, (const T *)tmp, x));
  count_launches(2);
  return PMG_OK;
}
template int sell_jacobi<float>(cudaStream_t, const Level &, const float *, float *, float *, double, int);
template int sell_jacobi<double>(cudaStream_t, const Level &, const double *, double *, double *, double, int);

template <typename T, int MODE>
static cudaError_t launch_gs(cudaStream_t s, const Level &L, int s0, int s1, const T *f, T *x, T omega, int num_sms) {
  // at most 8 warps per slice in FP32, 16 in FP64: the short colours of
  // levels 2-3 (42 and 318 slices), measured on the 64^3 bench: FP32
  // V-cycle 3.69 -> 3.61 ms with 8 (4: 3.96 ms); FP64 V-cycle 5.18 ->
  // 5.57 ms with 8
  const int k = pick_k(s1 - s0, num_sms, sizeof(T) == 4 ? 8 : 16);
#define PMG_GS(K_)                                                                                              \
  launch_pdl(k_sell_gs<T, K_, MODE>, dim3(slice_grid<T>(s1 - s0, num_sms, K_)), dim3(32 * K_), 0, s, s0, s1,     \
             (const int *)L.sell_perm.p, (const int *)L.sell_ptr.p, (const int *)L.sell_nlow.p,                  \
             (const int *)L.sell_col.p, (const short *)L.sell_c16.p, (const unsigned char *)L.sell_wide.p,       \
             sell_val<T>(L), sell_invd<T>(L), f, x, sell_sum<T>(L, false), sell_sum<T>(L, true), omega)
  return k == 16 ? PMG_GS(16) : k == 8 ? PMG_GS(8) : k == 4 ? PMG_GS(4) : PMG_GS(2);
#undef PMG_GS
}

// --------------------------------------------------------------- phases of an SSOR step
// What a phase's rows take from outside their blocks, over the whole GPU: the
// slices of the phase are consecutive, and nothing they read changes during
// the phase, so this is a product over a part of the matrix.  Leaves in
// base (slice order) f minus the outside part, and the outside sums in sl / su
// (see k_sell_gs for the sums):
//   GS_LOWER       base = f - lower_out,  sl = lower_out
//   GS_UPPER       base = f - upper_out,  su = upper_out
//   GS_FULL        base = f - lower_out,  sl = lower_out,  su = upper (all of it, from the old x)
// Bound by HBM on the finest level (values and column deltas once), by latency
// on the small ones.
template <typename T, int K, int MODE>
__global__ void __launch_bounds__(32 * K) k_sell_phase(int s0, int s1, const int *__restrict__ perm,
                                                       const int *__restrict__ sptr, const int *__restrict__ nlow,
                                                       const int *__restrict__ in, const int *__restrict__ col,
                                                       const short *__restrict__ c16,
                                                       const unsigned char *__restrict__ wide,
                                                       const T *__restrict__ val, const T *__restrict__ f,
                                                       const T *__restrict__ x, T *__restrict__ sl, T *__restrict__ su,
                                                       T *__restrict__ base) {
  constexpr int PF = 8;  // column steps per chunk
  constexpr bool FULL = MODE == GS_FULL;
  __shared__ T part[K][32], part_up[FULL ? K : 1][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int s = s0 + blockIdx.x;
  int off = 0, n = 0, nl = 0, gap = 0, r = -1;  // n steps; step j sits at j, or at j + gap from j = nl on (FULL)
  bool wd = false;
  int ci[PF];
  T cv[PF];
  auto load_chunk = [&](int c0) {
#pragma unroll
    for (int u = 0; u < PF; u++) {
      const int j = w + (c0 + u) * K, p = off + 32 * (FULL && j >= nl ? j + gap : j) + lane;
      if (wd) ci[u] = j < n ? __ldcs(col + p) : 0;
      else ci[u] = j < n ? (int)__ldcs(c16 + p) : 0;
      cv[u] = j < n ? __ldcs(val + p) : (T)0;
    }
  };
  auto start = [&](int q) {
    off = __ldg(sptr + q);
    n = (__ldg(sptr + q + 1) - off) >> 5;
    const int low = __ldg(nlow + q), ins = __ldg(in + q), li = ins & 0xffff, ui = ins >> 16;
    nl = low - li;
    if (MODE == GS_UPPER) {
      off += 32 * (low + 1 + ui);
      n -= low + 1 + ui;
    } else if (FULL) {
      gap = li + 1;
      n -= gap;
    } else {
      n = nl;
    }
    wd = __ldg(wide + q) != 0;
    r = __ldg(perm + q * 32 + lane);
    load_chunk(0);
  };
  if (s < s1) start(s);
  pdl_wait();
  pdl_trigger();
  for (; s < s1; s += gridDim.x) {
    const T *xb = wd ? x : x + (r > 0 ? r : 0);
    const T rest = w == 0 && r >= 0 ? __ldg(f + r) : (T)0;
    const int pos = s * 32 + lane;
    T sum = 0, up = 0;
    for (int c0 = 0;; c0 += PF) {
#pragma unroll
      for (int u = 0; u < PF; u++) {
        const int j = w + (c0 + u) * K;
        if (j < n) {
          const T t = cv[u] * __ldg(xb + ci[u]);
          if (!FULL || j < nl) sum += t;
          else up += t;
        }
      }
      if (w + (c0 + PF) * K >= n) break;
      load_chunk(c0 + PF);
    }
    part[w][lane] = sum;
    if (FULL) part_up[FULL ? w : 0][lane] = up;
    const int rr = r;
    const int sn = s + gridDim.x;
    if (sn < s1) start(sn);  // next slice's first chunk before the reduction
    __syncthreads();
    if (w == 0 && rr >= 0) {
#pragma unroll
      for (int k = 1; k < K; k++) {
        sum += part[k][lane];
        if (FULL) up += part_up[FULL ? k : 0][lane];
      }
      base[pos] = rest - sum;
      if (MODE == GS_UPPER) su[pos] = sum;
      else sl[pos] = sum;
      if (FULL) su[pos] = up;
    }
    __syncthreads();
  }
}

// The phase's own updates: one CTA per block goes through the phase's colours,
// forward, backward, or one after the other where the sweeps turn (the last
// phase of the forward sweep is the first one of the backward sweep and nothing
// lies between them).  A colour needs the block's earlier colours of this very
// launch only: they are kept in shared memory, addressed by 16-bit slots -- a few
// hundred cycles per colour instead of the 2.5-4 us of a launch.  What bounds it
// is latency and the instructions around it: a warp's work is a chain of tasks,
// one slice each, dealt out over the warps in the order of the colours, and all
// that a task needs to know is put into one 16-byte word of shared memory before
// the launch waits for its predecessor; the matrix steps (16-byte loads from a copy
// of the inside entries laid out for that) and vector entries of a warp's next
// task are on their way while other warps are at the colours in between.  The
// colours are kept apart by one counter each, to which the colour's slices add
// when they are done, and not by CTA barriers, which a warp busy with its loads
// would hold up.  (A wait ends because the earliest unfinished task never waits
// for a later one; it is bounded all the same.)
template <typename T>
struct BlkArgs {
  const int *tab;   // per block: first slice in meta / rows, first ordinal of every colour, number of slices
  const int4 *meta; // per slice: first chunk of its inside steps, counts (12 + 12 bits) and colour, slice
  const int *rows;  // 32 per slice
  int ncol, slots;
  const unsigned short *loc;
  const T *val, *invd, *f, *base;
  T *x, *sl, *su;
  T omega;
  int *err;
  int extra;  // added to what every wait expects (PMG_TEST_BLK_EXTRA)
};

// four steps of a lane: values and slots
template <typename T> struct BlkChunk;
template <> struct BlkChunk<float> {
  float4 v;
  uint2 c;
  __device__ __forceinline__ void zero() {
    v = make_float4(0.f, 0.f, 0.f, 0.f);
    c = make_uint2(0u, 0u);
  }
  __device__ __forceinline__ void load(const float *val, const unsigned short *loc, unsigned i) {
    v = __ldcs(reinterpret_cast<const float4 *>(val) + i);
    c = __ldcs(reinterpret_cast<const uint2 *>(loc) + i);
  }
  __device__ __forceinline__ float dot(const float *xs) const {
    const float x0 = xs[c.x & 0xffff], x1 = xs[c.x >> 16], x2 = xs[c.y & 0xffff], x3 = xs[c.y >> 16];
    return (v.x * x0 + v.y * x1) + (v.z * x2 + v.w * x3);
  }
};
template <> struct BlkChunk<double> {
  double2 v, u;
  uint2 c;
  __device__ __forceinline__ void zero() {
    v = u = make_double2(0.0, 0.0);
    c = make_uint2(0u, 0u);
  }
  __device__ __forceinline__ void load(const double *val, const unsigned short *loc, unsigned i) {
    v = __ldcs(reinterpret_cast<const double2 *>(val) + 2 * (size_t)i);
    u = __ldcs(reinterpret_cast<const double2 *>(val) + 2 * (size_t)i + 1);
    c = __ldcs(reinterpret_cast<const uint2 *>(loc) + i);
  }
  __device__ __forceinline__ double dot(const double *xs) const {
    const double x0 = xs[c.x & 0xffff], x1 = xs[c.x >> 16], x2 = xs[c.y & 0xffff], x3 = xs[c.y >> 16];
    return (v.x * x0 + v.y * x1) + (u.x * x2 + u.y * x3);
  }
};

// DIR: 1 forward, 2 backward.  TURN: a second pass in the other direction.
// SRC: what is left of f and of the outside sums before the first pass:
//   0: base, less the kept sums of the other side;  1: f, less the kept sums (after
//   a pass in the other direction of the same phase);  2: f (x = 0, first phase);
//   3: base (x = 0, the other phases).
// PLAIN: omega = 1; the colour at the turn has then just been updated and is left out.
// W warps; NC chunks of a task are held in registers, longer rows load the rest
// as they go (24 lower or higher neighbours in a plane of the Q2 / P2 lattices are 6 chunks).
template <typename T, int W, int NC, int DIR, bool TURN, int SRC, bool PLAIN>
__global__ void __launch_bounds__(32 * W, 1) k_sell_block(const __grid_constant__ BlkArgs<T> a) {
  constexpr int SECOND = 1 << 30, NO_DEP = 255;
  extern __shared__ __align__(16) unsigned char blk_sm[];
  T *xs = reinterpret_cast<T *>(blk_sm);
  T *ks = xs + a.slots;  // TURN: f less pass 0's side, what pass 1 starts from
  // first chunk | chunks (12 bits), hop (8), hop to wait for (8), second pass | position | slot
  int4 *task = reinterpret_cast<int4 *>(ks + (TURN ? a.slots : 0));
  __shared__ int tab[BLK_MAX_COLOURS + 2], dep[2 * BLK_MAX_COLOURS], need[2 * BLK_MAX_COLOURS];
  __shared__ int done[2 * BLK_MAX_COLOURS];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, ncol = a.ncol;
  if (threadIdx.x < ncol + 2) tab[threadIdx.x] = __ldg(a.tab + (size_t)blockIdx.x * (ncol + 2) + threadIdx.x);
  for (int i = threadIdx.x; i < a.slots; i += 32 * W) xs[i] = (T)0;
  __syncthreads();
  const int m0 = tab[0], ns = tab[1 + ncol];
  // hops: pass 0 over all colours, pass 1 without its first one if PLAIN
  const int hops = TURN ? 2 * ncol - PLAIN : ncol;
  if (threadIdx.x < hops) {
    auto slices = [&](int h) {
      const bool fwd = (h < ncol) == (DIR == 1);
      const int k = h < ncol ? h : h - ncol + PLAIN, c = fwd ? k : ncol - 1 - k;
      return tab[2 + c] - tab[1 + c];
    };
    const int h = threadIdx.x;
    int p = h - 1;
    while (p >= 0 && slices(p) == 0) p--;
    dep[h] = p < 0 ? NO_DEP : p;
    need[h] = slices(h) + a.extra;
    done[h] = 0;
  }
  __syncthreads();
  // tasks: the slices of pass 0 in order, then those of pass 1
  const int skip1 = !PLAIN ? 0 : DIR == 2 ? tab[2] : ns - tab[ncol];  // slices left out at the turn
  const int total = TURN ? 2 * ns - skip1 : ns;
  for (int i = threadIdx.x; i < ns; i += 32 * W) {
    const int4 m = __ldg(a.meta + m0 + i);
    const int li = ((m.y & 0xfff) + 3) >> 2, ui = ((m.y >> 12 & 0xfff) + 3) >> 2, c = m.y >> 24;
    int h = DIR == 1 ? c : ncol - 1 - c;
    task[DIR == 1 ? i : ns - 1 - i] =
        make_int4(m.x + (DIR == 1 ? 0 : li), (DIR == 1 ? li : ui) | h << 12 | dep[h] << 20, m.z * 32, i * 32);
    if (TURN) {
      const int q = (DIR == 2 ? i : ns - 1 - i) - skip1;
      h = (DIR == 2 ? c : ncol - 1 - c) + ncol - PLAIN;
      if (q >= 0)
        task[ns + q] = make_int4(m.x + (DIR == 2 ? 0 : li), (DIR == 2 ? li : ui) | h << 12 | dep[h] << 20 | SECOND,
                                 m.z * 32, i * 32);
    }
  }
  __syncthreads();
  T *const sum0 = DIR == 1 ? a.sl : a.su, *const sum1 = DIR == 1 ? a.su : a.sl;  // left by pass 0 / pass 1
  const int *rows = a.rows + (size_t)m0 * 32 + lane;
  BlkChunk<T> ch[NC];
  T id = 0, r0 = 0, r1 = 0, ro = 0;  // 1 / a_rr; base or f; kept sum of the other side; own outside sum
  int4 t = make_int4(0, 0, 0, 0);
  int row = -1;
  auto fetch_matrix = [&](int g) {
    t = task[g];
    row = __ldg(rows + t.w);
    id = __ldg(a.invd + t.z + lane);
    const int n = t.y & 0xfff;
    const unsigned at = (unsigned)t.x * 32 + lane;
#pragma unroll
    for (int u = 0; u < NC; u++) {
      ch[u].zero();
      if (u < n) ch[u].load(a.val, a.loc, at + 32 * u);
    }
  };
  auto fetch_vectors = [&]() {
    if (TURN && t.y & SECOND) return;
    const int pos = t.z + lane;
    if (SRC == 0 || SRC == 3) {
      r0 = a.base[pos];
      ro = sum0[pos];
    } else {
      r0 = a.f[row < 0 ? 0 : row];
    }
    if (SRC < 2) r1 = sum1[pos];
  };
  bool failed = false;
  if (w < total) fetch_matrix(w);
  pdl_wait();
  pdl_trigger();
  if (w < total) fetch_vectors();
  const unsigned done0 = (unsigned)__cvta_generic_to_shared(done);
  for (int g = w; g < total; g += W) {
    const bool second = TURN && t.y & SECOND;
    const int n = t.y & 0xfff, hop = t.y >> 12 & 0xff, d = t.y >> 20 & 0xff, pos = t.z + lane;
    if (d != NO_DEP) {
      const int want = need[d];
      for (int it = 0; !failed; it++) {
        int got;
        asm volatile("ld.acquire.cta.shared::cta.s32 %0, [%1];" : "=r"(got) : "r"(done0 + 4 * d) : "memory");
        if (got >= want) break;
        if (it > (1 << 23)) {  // about 0.2 s
          failed = true;
          atomicExch(a.err, 1);
        }
      }
    }
    T sum = 0;
#pragma unroll
    for (int u = 0; u < NC; u++) sum += ch[u].dot(xs);
    for (int u = NC; u < n; u++) {
      BlkChunk<T> c;
      c.load(a.val, a.loc, (unsigned)t.x * 32 + lane + 32 * u);
      sum += c.dot(xs);
    }
    if (row >= 0) {
      const T rest = second ? ks[t.w + lane] : r0 - r1;
      T v = (rest - sum) * id;
      if (!PLAIN) {
        const T xr = a.x[row];
        v = xr + a.omega * (v - xr);
      }
      xs[t.w + lane] = v;
      if (TURN && !second) ks[t.w + lane] = r0 - sum;
      (second ? sum1 : sum0)[pos] = second ? sum : ro + sum;
      a.x[row] = v;
    }
    __syncwarp();
    if (lane == 0)
      asm volatile("red.release.cta.shared::cta.add.s32 [%0], 1;" ::"r"(done0 + 4 * hop) : "memory");
    if (g + W < total) {
      fetch_matrix(g + W);
      fetch_vectors();
    }
  }
}

template <typename T>
static T *sell_base(const Level &L) {
  if (sizeof(T) == 4) return reinterpret_cast<T *>(L.sell_base32.p);
  return reinterpret_cast<T *>(L.sell_base64.p);
}

// shared memory of a phase's block kernel: iterate and tasks, for two passes also
// what the second one starts from
template <typename T>
static size_t blk_smem(const Level &L, int p, bool turn) {
  return (turn ? 2 : 1) * ((size_t)L.blk_slots[p] * sizeof(T) + (size_t)(L.blk_slots[p] / 32) * BLK_TASK);
}

// whether the level's SSOR sweeps run by blocks in this precision
template <typename T>
static bool use_blocks(const Level &L) {
  return L.blk_on[sizeof(T) == 8];
}

// What the sweeps need beside the values: the kept sums and, for SSOR steps by
// blocks, the base vector and the blocks' copy of the entries inside them.  Products
// need none of it (the FP64 finest matrix of an FP32 V-cycle: at Q2 64^3 0.4 GB and a
// pass over the matrix per solve).
template <typename T>
int sell_sweep_values(Handle &h, Level &L, bool ssor) {
  const bool f32 = sizeof(T) == 4;
  PMG_TRY(sell_values<T>(h, L));
  if (f32) PMG_TRY(alloc_sums(h, L, L.sums_mem32, L.sell_sl32, L.sell_su32));
  else PMG_TRY(alloc_sums(h, L, L.sums_mem64, L.sell_sl64, L.sell_su64));
  if (!ssor || !use_blocks<T>(L) || (f32 ? L.blk_val_fresh32 : L.blk_val_fresh64)) return PMG_OK;
  const size_t rows = (size_t)L.sell_nslices * 32, nval = (size_t)L.blk_chunks * 128;
  Carve parts;
  if (f32) parts.add(L.sell_base32, rows), parts.add(L.blk_val32, nval);
  else parts.add(L.sell_base64, rows), parts.add(L.blk_val64, nval);
  PMG_TRY(parts.place(f32 ? L.blk_mem32 : L.blk_mem64));
  T *bval = f32 ? reinterpret_cast<T *>(L.blk_val32.p) : reinterpret_cast<T *>(L.blk_val64.p);
  const int n = (int)(L.blk_meta.n / 4);
  k_blk_values<T><<<std::min((n + 7) / 8, h.num_sms * 16), 256, 0, h.stream>>>(
      n, reinterpret_cast<const int4 *>(L.blk_meta.p), L.sell_ptr.p, L.sell_nlow.p, sell_val<T>(L), bval);
  count_launches(1);
  PMG_CUDA(cudaGetLastError());
  if (f32) L.blk_val_fresh32 = true;
  else L.blk_val_fresh64 = true;
  return PMG_OK;
}
template int sell_sweep_values<float>(Handle &, Level &, bool);
template int sell_sweep_values<double>(Handle &, Level &, bool);

template <typename T, int MODE>
static int launch_phase(cudaStream_t st, const Level &L, int p, const T *f, const T *x, int num_sms) {
  const int s0 = L.sell_group[L.blk_col[p]], s1 = L.sell_group[L.blk_col[p + 1]];
  const int k = std::max(4, pick_k(s1 - s0, num_sms));
#define PMG_PHASE(K_)                                                                                            \
  launch_pdl(k_sell_phase<T, K_, MODE>, dim3(slice_grid<T>(s1 - s0, num_sms, K_)), dim3(32 * K_), 0, st, s0, s1,  \
             (const int *)L.sell_perm.p, (const int *)L.sell_ptr.p, (const int *)L.sell_nlow.p,                   \
             (const int *)L.sell_in.p, (const int *)L.sell_col.p, (const short *)L.sell_c16.p,                    \
             (const unsigned char *)L.sell_wide.p, sell_val<T>(L), f, x, sell_sum<T>(L, false),                   \
             sell_sum<T>(L, true), sell_base<T>(L))
  PMG_CUDA((k == 16 ? PMG_PHASE(16) : k == 8 ? PMG_PHASE(8) : PMG_PHASE(4)));
#undef PMG_PHASE
  count_launches(1);
  return PMG_OK;
}

template <typename T, int W, int NC, int DIR, bool TURN, int SRC, bool PLAIN>
static int launch_block_k(cudaStream_t st, const BlkArgs<T> &a, int blocks, size_t smem) {
  PMG_CUDA(func_smem(k_sell_block<T, W, NC, DIR, TURN, SRC, PLAIN>, BLK_SMEM));
  PMG_CUDA(launch_pdl(k_sell_block<T, W, NC, DIR, TURN, SRC, PLAIN>, dim3(blocks), dim3(32 * W), smem, st, a));
  count_launches(1);
  return PMG_OK;
}

template <typename T, int DIR, bool TURN, int SRC>
static int launch_block(cudaStream_t st, const Level &L, int p, const T *f, T *x, T omega, int *err) {
  const size_t smem = blk_smem<T>(L, p, TURN);
  if (TURN && smem > BLK_SMEM) {
    // no room for both passes: one launch each, the second one from f again
    PMG_TRY((launch_block<T, DIR, false, SRC>(st, L, p, f, x, omega, err)));
    return launch_block<T, 3 - DIR, false, 1>(st, L, p, f, x, omega, err);
  }
  BlkArgs<T> a{};
  a.tab = L.blk_tab.p + L.blk_tab0[p];
  a.meta = reinterpret_cast<const int4 *>(L.blk_meta.p);
  a.rows = L.blk_rows.p;
  a.ncol = L.blk_col[p + 1] - L.blk_col[p];
  a.slots = L.blk_slots[p];
  a.loc = L.sell_loc.p;
  a.val = sizeof(T) == 4 ? reinterpret_cast<const T *>(L.blk_val32.p) : reinterpret_cast<const T *>(L.blk_val64.p);
  a.invd = sell_invd<T>(L);
  a.f = f;
  a.base = sell_base<T>(L);
  a.x = x;
  a.sl = sell_sum<T>(L, false);
  a.su = sell_sum<T>(L, true);
  a.omega = omega;
  a.err = err;
  // PMG_TEST_BLK_EXTRA=<n>: every wait expects n slices that nobody does, so it runs
  // out -- the test of the give-up path (read at every launch; a captured V-cycle
  // graph keeps the value it was captured with)
  const char *extra = getenv("PMG_TEST_BLK_EXTRA");
  a.extra = extra ? std::max(0, atoi(extra)) : 0;
  const int nb = L.blk_n[p];
  // 16 warps with every row's chunks in registers while a block has few slices,
  // and in FP64 always (registers); 32 warps with 4 chunks for the larger blocks
  // in FP32.  Measured on the 64^3 Q2 levels, one pass over 9 colours: 36 slices
  // 4.3 us (32 warps: 7.3), 126 slices 8.6 us (16 warps: 10.0), 522 slices 24 us;
  // FP64 V-cycle of the 32^3 Q2 hierarchy 1.25 ms (32 warps: 1.37)
#define PMG_BLK(W_, NC_)                                                                                   \
  (omega == (T)1 ? launch_block_k<T, W_, NC_, DIR, TURN, SRC, true>(st, a, nb, smem)                         \
                 : launch_block_k<T, W_, NC_, DIR, TURN, SRC, false>(st, a, nb, smem))
  if (sizeof(T) == 8 || L.blk_slots[p] / 32 <= 64) return PMG_BLK(16, 6);
  return PMG_BLK(32, 4);
#undef PMG_BLK
}

// one SSOR sweep by colours: forward (sides: GS_LOWER / GS_LOWER_ZERO /
// GS_FULL) or backward (GS_UPPER, GS_FULL); the first `skip` colours are left out
template <typename T>
static int sweep_colours(cudaStream_t s, const Level &L, bool forward, int mode, int skip, const T *f, T *x, T omega,
                         int num_sms) {
  const int nc = (int)L.sell_group.size() - 2;
  for (int cc = skip; cc < nc; cc++) {
    const int c = forward ? cc : nc - 1 - cc;
    const int s0 = L.sell_group[c], s1 = L.sell_group[c + 1];
    if (s1 <= s0) continue;
    PMG_CUDA((mode == GS_FULL    ? launch_gs<T, GS_FULL>(s, L, s0, s1, f, x, omega, num_sms)
              : mode == GS_UPPER ? launch_gs<T, GS_UPPER>(s, L, s0, s1, f, x, omega, num_sms)
              : mode == GS_LOWER ? launch_gs<T, GS_LOWER>(s, L, s0, s1, f, x, omega, num_sms)
                                 : launch_gs<T, GS_LOWER_ZERO>(s, L, s0, s1, f, x, omega, num_sms)));
    count_launches(1);
  }
  return PMG_OK;
}

// SSOR steps (TMGLevel3D::SSOR in colour order): forward over the colours, then
// backward, `steps` times; x_D = f_D holds already and stays.  With omega = 1 a
// Gauss-Seidel update of a colour directly after an update of the same colour
// leaves x unchanged (the colour's rows have zero residual and are not coupled
// to each other), so the second of two successive updates of a colour is left
// out where the sweeps turn.  (The skipped passes' sums stay right: the last
// colour has no higher colours and the first no lower ones, so theirs are
// always 0.)  Where two rows of one colour are coupled (sell_coupled) a repeated
// update does change x, and none is left out.
//
// By blocks (where block_gain says so), one phase is a product over the whole GPU
// for what comes from outside and one launch for the phase's own colours: 27 colours
// in 3 phases are 10 launches for a step on an arbitrary x, 9 from x = 0 and 8 after
// another step, instead of 53 (52 after another step).  Measured (64^3 Q2 hierarchy,
// FP32 / FP64 V-cycle): one launch per colour over whole rows 3.60 / 4.71 ms, over the
// split rows 3.4 / 4.5, by blocks 2.25 / 3.56, by blocks but for the finest FP64 level
// 3.09.  On the finest level (2.1 M rows) a phase takes 31-51 us for the outside part (100 / 200 MB; 3.5-3.9 TB/s, bound by the
// latency of short rows) and 24 us for its 9 colours (43 planes on 43 SMs); on
// the 36 k-row level 3.5 + 4.3 us, where 9 colour launches took 23 us.
template <typename T>
int sell_ssor(cudaStream_t s, const Level &L, const T *f, T *x, double omega, int num_sms, int steps, SweepStart start,
              int *err) {
  const T om = (T)omega;
  if (!use_blocks<T>(L)) {
    const int skip = omega == 1.0 && !L.sell_coupled ? 1 : 0;
    for (int k = 0; k < steps; k++) {
      const int fwd = !L.sell_split || (k == 0 && start == SWEEP_ANY) ? GS_FULL
                      : k == 0                                        ? GS_LOWER_ZERO
                                                                      : GS_LOWER;
      PMG_TRY(sweep_colours<T>(s, L, true, fwd, k > 0 ? skip : 0, f, x, om, num_sms));
      PMG_TRY(sweep_colours<T>(s, L, false, L.sell_split ? GS_UPPER : GS_FULL, skip, f, x, om, num_sms));
    }
    return PMG_OK;
  }
  const int P = (int)L.blk_col.size() - 1;
  for (int k = 0; k < steps; k++) {
    const bool any = k == 0 && start == SWEEP_ANY, zero = k == 0 && !any;
    // forward; the first phase needs nothing from outside unless x is arbitrary,
    // and after a backward sweep it has run with that sweep's last phase
    if (any) {
      PMG_TRY((launch_phase<T, GS_FULL>(s, L, 0, f, x, num_sms)));
      PMG_TRY((launch_block<T, 1, false, 0>(s, L, 0, f, x, om, err)));
    } else if (zero) {
      PMG_TRY((launch_block<T, 1, false, 2>(s, L, 0, f, x, om, err)));
    }
    for (int p = 1; p < P; p++) {
      if (any) PMG_TRY((launch_phase<T, GS_FULL>(s, L, p, f, x, num_sms)));
      else PMG_TRY((launch_phase<T, GS_LOWER>(s, L, p, f, x, num_sms)));
      if (zero && p == P - 1) PMG_TRY((launch_block<T, 1, true, 3>(s, L, p, f, x, om, err)));
      else if (zero) PMG_TRY((launch_block<T, 1, false, 3>(s, L, p, f, x, om, err)));
      else if (p == P - 1) PMG_TRY((launch_block<T, 1, true, 0>(s, L, p, f, x, om, err)));
      else PMG_TRY((launch_block<T, 1, false, 0>(s, L, p, f, x, om, err)));
    }
    for (int p = P - 2; p >= 0; p--) {
      PMG_TRY((launch_phase<T, GS_UPPER>(s, L, p, f, x, num_sms)));
      if (p == 0 && k + 1 < steps) PMG_TRY((launch_block<T, 2, true, 0>(s, L, p, f, x, om, err)));
      else PMG_TRY((launch_block<T, 2, false, 0>(s, L, p, f, x, om, err)));
    }
  }
  return PMG_OK;
}
template int sell_ssor<float>(cudaStream_t, const Level &, const float *, float *, double, int, int, SweepStart, int *);
template int sell_ssor<double>(cudaStream_t, const Level &, const double *, double *, double, int, int, SweepStart, int *);

// one SOR step (TMGLevel3D::SOR, MGLevel3D.C:280-361): the forward sweep alone,
// over whole rows (the next step's higher colours hold new values)
template <typename T>
int sell_sor(cudaStream_t s, const Level &L, const T *f, T *x, double omega, int num_sms) {
  return sweep_colours<T>(s, L, true, GS_FULL, 0, f, x, (T)omega, num_sms);
}
template int sell_sor<float>(cudaStream_t, const Level &, const float *, float *, double, int);
template int sell_sor<double>(cudaStream_t, const Level &, const double *, double *, double, int);

}  // namespace pmg
