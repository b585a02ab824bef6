// resident.cuh -- the middle steps of a run of spheres among static obstacles on
// resident pair lists (included by kernels.cuh, in namespace gg).
//
// The launched pipeline lists every particle's contacts anew in every step:
// three sort kernels, the 27-cell walk, the search of the partner's list entry
// and of the pair's memory row.  Here the pairs whose surfaces are closer than a
// skin are listed once and kept until a particle has moved half the skin, so a
// pair that is not listed cannot have met.  A step is then three launches:
//
//   res_rebuild_kernel  (returns at once unless a particle has moved half the
//                       skin) cell lists of the current positions, pair lists,
//                       contact memory carried over
//   res_pairs_kernel    every listed pair's exact overlap test, the contact law
//                       of those in contact with the memory in the pair's slot,
//                       both sides' results; the obstacle candidates; the
//                       candidate-pair count of the step
//   res_sums_kernel     per-particle sums in the order of the launched pipeline
//                       (cell of the partner, then id; obstacles last), kicks,
//                       drift, cell key and count, the obstacle candidates of
//                       the new position, the displacement check
//
// The results are those of the launched pipeline to the bit: the same contacts
// (the exact test runs on every listed pair in every step), the same law with
// the same operands, the same order of sums, the same status bits and counts.
// The last step of every call runs the launched pipeline, which leaves contact
// lists, memory rows and coordination as before.

// control words
enum {
  kResRequest = 0, kResFailed = 1, kResRowPairs = 2, kResValid = 3, kResObs = 4, kResCountAll = 6
};
// kResRequest: 0 lists are good, 1 a particle has moved half the skin, other
// values: first build of a run (the memory rows are current)
// kResFailed: the contacts did not fit in the lists; the run stands still from
// that step on.  kResRowPairs: the rows hold the pairs' memories, not the
// obstacles' (a rebuild that has not ended).  kResValid: pairs of a complete build,
// else -1; kResObs, kResObs + 1: obstacle items of the steps of even and odd
// parity; kResCountAll: the step's candidate pairs are counted over all cells, not
// from the step before

// the state of a listed pair or of a particle's obstacle
enum { kResContact = 1, kResMemory = 2, kResCandidate = 4 };

// force and torque of one side of a listed pair: one 32-byte sector in mixed precision
template <typename R>
struct ResResult {
  typename Vec4<R>::type f;  // w: 0 no contact; a contact: 1 the partner owns it, else 2, with a memory 3
  typename Vec4<R>::type t;
};

template <typename R>
__device__ __forceinline__ PairMemory<R> res_load_memory(const R* m, size_t stride, bool rolling) {
  PairMemory<R> x;
  x.kdelta = v3<R>(m[0], m[stride], m[2 * stride]);
  x.prev_normal = v3<R>(m[3 * stride], m[4 * stride], m[5 * stride]);
  // without a rolling spring the stored one stays where it is
  x.spring = rolling ? v3<R>(m[6 * stride], m[7 * stride], m[8 * stride]) : v3<R>(R(0), R(0), R(0));
  return x;
}
template <typename R>
__device__ __forceinline__ void res_store_memory(R* m, size_t stride, const PairMemory<R>& x, bool spring) {
  m[0] = x.kdelta.x;
  m[stride] = x.kdelta.y;
  m[2 * stride] = x.kdelta.z;
  m[3 * stride] = x.prev_normal.x;
  m[4 * stride] = x.prev_normal.y;
  m[5 * stride] = x.prev_normal.z;
  if (spring) {
    m[6 * stride] = x.spring.x;
    m[7 * stride] = x.spring.y;
    m[8 * stride] = x.spring.z;
  }
}

// ---- the lists ------------------------------------------------------------------

// Lanes that share a particle in a build: they take a row's candidates and a
// list's entries side by side.  One thread per particle walked some 60 candidates
// twice in a chain of dependent loads (1,000 spheres: 0.27 ms a build, 0.15 with
// the lanes; 200,000: 0.46 -> 0.32 ms).  Eight lanes are as fast on dense beds
// but idle on sparse rows (410,000 falling spheres: 0.40 against 0.30 ms).
constexpr int kResLanes = 4;
constexpr int kResRows = 16;  // rows of cells a walk can meet
__device__ __forceinline__ int res_lane() { return threadIdx.x & (kResLanes - 1); }
__device__ __forceinline__ int res_group_shift() { return (threadIdx.x & 31) & ~(kResLanes - 1); }
// the group's lanes for which b holds (every lane of the warp calls it)
__device__ __forceinline__ unsigned res_ballot(bool b) {
  return (__ballot_sync(0xffffffffu, b) >> res_group_shift()) & ((1u << kResLanes) - 1u);
}

// put(hit, entry, own) in rounds of kResLanes lanes, in the order of (cell, id), for
// every particle whose surface is closer than `skin` to that of particle s.  The
// cells that hold such particles: every centre within r_s + r_max + skin, at most
// 4 x 4 rows of cells (the cells are no smaller than the largest diameter).
// Every lane of the warp calls it; active: the group has a particle; range: shared
// memory of the group.
template <typename R, typename F>
__device__ __forceinline__ void res_walk(const StepArgs<R>& a, const ResArgs<R>& r, int s, bool active, double skin,
                                         int2* range, F put) {
  const unsigned full = 0xffffffffu;
  const int lane = res_lane();
  double4 xi = make_double4(0., 0., 0., 0.);
  int id = 0, rows = 0;
  if (active) {
    xi = a.cur.xr[s];
    const int4 mi = a.cur.meta[s];
    id = mi.x;
    const SysDev& S = a.sys[mi.w];
    const double reach = (xi.w + r.r_max[mi.w] + skin) * (1. + 1.e-9);
    auto cell = [](double x, double o, double e, int n) { return min(max((int)floor((x - o) / e), 0), n - 1); };
    const int i0 = cell(xi.x - reach, S.ox, S.ex, S.nbi), i1 = cell(xi.x + reach, S.ox, S.ex, S.nbi);
    const int j0 = cell(xi.y - reach, S.oy, S.ey, S.nbj), j1 = cell(xi.y + reach, S.oy, S.ey, S.nbj);
    const int k0 = cell(xi.z - reach, S.oz, S.ez, S.nbk), k1 = cell(xi.z + reach, S.oz, S.ez, S.nbk);
    const int nk = k1 - k0 + 1;
    rows = min((j1 - j0 + 1) * nk, kResRows);
    for (int row = lane; row < rows; row += kResLanes) {
      const int j = j0 + row / nk, k = k0 + row % nk;
      range[row] = make_int2(a.cell_start[cell_index(S, i0, j, k)], a.cell_start[cell_index(S, i1, j, k) + 1]);
    }
  }
  __syncwarp();
  for (int row = 0; __any_sync(full, row < rows); row += 2) {
    int b[2], e[2], t[2];
    double4 xj[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int2 be = row + u < rows ? range[row + u] : make_int2(0, 0);
      b[u] = be.x;
      e[u] = be.y;
      t[u] = b[u] + lane < e[u] ? a.perm[b[u] + lane] : -1;
    }
#pragma unroll
    for (int u = 0; u < 2; ++u)
      if (t[u] >= 0) xj[u] = a.cur.xr[t[u]];
#pragma unroll
    for (int u = 0; u < 2; ++u)
      for (int q = b[u];;) {
        bool hit = false, own = false;
        if (t[u] >= 0 && t[u] != s) {
          const double dx = xj[u].x - xi.x, dy = xj[u].y - xi.y, dz = xj[u].z - xi.z;
          // symmetric: both sides list the pair; with the margin every contact even without a skin
          const double rs = (xi.w + xj[u].w) * (1. + 1.e-12) + skin;
          hit = dx * dx + dy * dy + dz * dz < rs * rs;
          own = hit && id < a.cur.meta[t[u]].x;
        }
        put(hit, t[u] | (own ? kOwnBit : 0), own);
        q += kResLanes;
        if (!__any_sync(full, q < e[u])) break;
        t[u] = q + lane < e[u] ? a.perm[q + lane] : -1;
        if (t[u] >= 0) xj[u] = a.cur.xr[t[u]];
      }
  }
}

// the memory of the listed pairs of particle s back into its memory row, by the
// lanes of a group (every lane of the warp calls it); returns the row's entries
template <typename R>
__device__ __forceinline__ int res_flush_pairs(const StepArgs<R>& a, const ResArgs<R>& r, int s, bool active) {
  const unsigned full = 0xffffffffu;
  const int lane = res_lane();
  const unsigned lower = (1u << lane) - 1u;
  int2 en = make_int2(0, 0);
  int row = 0, cnt = 0;
  if (active) {
    en = r.ent[s];
    row = a.cur.orig[s];
  }
  HistEntry<R>* h = a.hist_prev + (size_t)row * a.hist_cap;
  for (int q0 = 0; __any_sync(full, q0 < en.y); q0 += kResLanes) {
    const int e = q0 + lane < en.y ? r.nb[en.x + q0 + lane] : 0;
    const int mine = e & kOwnBit ? r.ent_pair[en.x + q0 + lane] : 0;
    const bool keep = (e & kOwnBit) && (r.state[mine] & kResMemory);
    const unsigned keepers = res_ballot(keep);
    const int at = cnt + __popc(keepers & lower);
    if (keep && at < a.hist_cap) {
      const PairMemory<R> m = res_load_memory(r.mem + mine, (size_t)r.pair_cap, true);
      HistEntry<R> x;
      x.other = a.cur.meta[entry_slot(e)].x;
      x.flags = 0;
      x.kd[0] = m.kdelta.x; x.kd[1] = m.kdelta.y; x.kd[2] = m.kdelta.z;
      x.n[0] = m.prev_normal.x; x.n[1] = m.prev_normal.y; x.n[2] = m.prev_normal.z;
      x.sp[0] = m.spring.x; x.sp[1] = m.spring.y; x.sp[2] = m.spring.z;
      h[at] = x;
    } else if (keep) {
      set_status(a.stats, GRAINS_GPU_HISTORY_FULL);
    }
    cnt += __popc(keepers);
  }
  cnt = min(cnt, a.hist_cap);
  if (active && lane == 0) a.hist_n_prev[row] = cnt;
  return cnt;
}

// what the HookeMemory law forms from the two bodies alone, with its own
// expressions (normal_part_fp64 of the mixed path, hooke_memory of the FP64 one:
// the same operations)
template <typename R>
__device__ __forceinline__ ResConst res_constants(const StepArgs<R>& a, int s, int t) {
  const int4 mi = a.cur.meta[s], mj = a.cur.meta[t];
  const double4 mdi = a.cur.md[s], mdj = a.cur.md[t];
  const SysDev& S = a.sys[mi.w];
  ResConst k;
  k.law = S.law_offset + mi.y * S.n_mat + mj.y;
  const LawParams<R>& L = a.laws[k.law];
  const double avmass = 1. / (1. / mdi.x + 1. / mdj.x);
  k.gamman = -2. * L.beta64 * std::sqrt(avmass * L.kn64);
  const double etat = L.etat64 == -1. ? -L.beta64 * std::sqrt(L.kn64 / avmass) : L.etat64;
  k.gammat = 2. * etat * avmass;
  k.crust = xadd(mdi.y, mdj.y);
  k.pad = 0;
  return k;
}

// One cooperative launch: the cell lists, the pair lists, the memory.  Every
// barrier wait is bounded (grid_barrier).  A build that gives up, at whichever
// barrier, leaves kResValid at -1, on which the other kernels do nothing, and the
// status bit, on which no later launch builds.
constexpr int kResHits = 64;  // a particle's listed partners kept in shared memory during its walk
template <typename R>
__global__ void __launch_bounds__(256, 3) res_rebuild_kernel(StepArgs<R> a, ResArgs<R> r, int step) {
  const int request = *(volatile int*)(r.ctl + kResRequest);
  if (request == 0) return;
  const int nthreads = gridDim.x * blockDim.x, tid = blockIdx.x * blockDim.x + threadIdx.x;
  if (*(volatile int*)(r.ctl + kResFailed) || (*(volatile int*)&a.stats->status & GRAINS_GPU_TIMEOUT)) {
    if (threadIdx.x == 0) r.ctl[kResValid] = -1;
    return;
  }
  // a test of the bounded waits: this block leaves a rebuild before its first barrier
  if (request == 1 && (int)blockIdx.x == a.barrier_skip_block) return;
  auto meet = [&]() {
    const bool ok = grid_barrier(r.bar, &a.stats->status, a.barrier_polls);
    if (!ok && threadIdx.x == 0) r.ctl[kResValid] = -1;
    return ok;
  };
  const int n = a.n, C = a.n_cells;
  const int* count = r.count[step % 3];
  __shared__ int offset_s;
  __shared__ int hit_s[256 / kResLanes][kResHits];
  __shared__ int2 range_s[256 / kResLanes][kResRows];
  int* hits = hit_s[threadIdx.x / kResLanes];
  int2* range = range_s[threadIdx.x / kResLanes];
  const int lane = res_lane();
  const unsigned lower = (1u << lane) - 1u;
  const int groups = nthreads / kResLanes, group = tid / kResLanes;
  const int padded = (n + groups - 1) / groups * groups;
  if (request == 1)
    for (int s = group; s < padded; s += groups) res_flush_pairs(a, r, s, s < n);
  // exclusive scan of the cell counts: a chunk per block, then the offsets
  const int chunk = (C + gridDim.x - 1) / gridDim.x;
  const int c0 = min(C, (int)blockIdx.x * chunk), c1 = min(C, c0 + chunk);
  int run = 0;
  for (int base = c0; base < c1; base += blockDim.x) {
    const int i = base + threadIdx.x;
    const int v = i < c1 ? count[i] : 0;
    int total;
    const int pre = block_exclusive_scan(v, &total);
    if (i < c1) a.cell_start[i] = run + pre;
    run += total;
  }
  if (threadIdx.x == 0) r.block_sums[blockIdx.x] = run;
  if (!meet()) return;
  if (tid == 0) {
    r.ctl[kResValid] = -1;
    if (request == 1) r.ctl[kResRowPairs] = 1;
    r.total[0] = r.total[1] = 0;
  }
  int part = 0;
  for (int b = threadIdx.x; b < (int)blockIdx.x; b += blockDim.x) part += r.block_sums[b];
  int before;
  block_exclusive_scan(part, &before);
  if (threadIdx.x == 0) {
    offset_s = before;
    if (blockIdx.x == gridDim.x - 1) a.cell_start[C] = before + run;
  }
  __syncthreads();
  for (int i = c0 + threadIdx.x; i < c1; i += blockDim.x) {
    const int v = a.cell_start[i] + offset_s;
    a.cell_start[i] = v;
    a.cell_cursor[i] = v;
  }
  if (!meet()) return;
  for (int s = tid; s < n; s += nthreads) scatter_one(a, s);
  if (!meet()) return;
  for (int c = tid; c < C; c += nthreads) cell_order(a, a.cell_start[c], a.cell_start[c + 1]);
  if (!meet()) return;
  // the lists, with half the skin again when they do not fit
  double skin = r.skin0;
  for (;;) {
    for (int s = group; s < padded; s += groups) {
      int cnt = 0, own = 0;
      res_walk(a, r, s, s < n, skin, range, [&](bool hit, int e, bool o) {
        const unsigned m = res_ballot(hit);
        const int at = cnt + __popc(m & lower);
        if (hit && at < kResHits) hits[at] = e;
        cnt += __popc(m);
        own += __popc(res_ballot(o));
      });
      __syncwarp();
      const bool leader = lane == 0;
      // in 64 bits: particles piled up count more than 2^31 entries before the lists are known not to fit
      unsigned long long e64 = warp_reserve(r.total, leader ? (unsigned long long)cnt : 0ull),
                         p64 = warp_reserve(r.total + 1, leader ? (unsigned long long)own : 0ull);
      e64 = __shfl_sync(0xffffffffu, e64, res_group_shift());
      p64 = __shfl_sync(0xffffffffu, p64, res_group_shift());
      const bool fits = e64 + cnt <= (unsigned long long)r.ent_cap && p64 + own <= (unsigned long long)r.pair_cap;
      const int e0 = fits ? (int)e64 : 0, p0 = fits ? (int)p64 : 0;
      if (s < n && leader) {
        r.ent[s] = make_int2(e0, fits ? cnt : 0);
        r.x0[s] = a.cur.xr[s];
        r.dirty[0][s] = r.dirty[1][s] = 0;
      }
      // entry q of the list; the pair of an owned one
      int q0 = 0, rank = 0;
      auto enter = [&](bool in, int e) {
        const bool o = in && (e & kOwnBit);
        const unsigned ins = res_ballot(in), owners = res_ballot(o);
        if (in) {
          const int q = e0 + q0 + __popc(ins & lower);
          r.nb[q] = e;
          r.res[q].f.w = R(0);
          if (o) {
            const int p = p0 + rank + __popc(owners & lower);
            r.pair[p] = make_int4(s, entry_slot(e), q, -1);
            r.ent_pair[q] = p;
          }
        }
        q0 += __popc(ins);
        rank += __popc(owners);
      };
      const bool kept = cnt <= kResHits || !fits;  // nothing is entered when it does not fit
      for (int q = 0; __any_sync(0xffffffffu, kept && fits && q < cnt); q += kResLanes) {
        const bool in = kept && fits && q + lane < cnt;
        enter(in, in ? hits[q + lane] : 0);
      }
      if (__any_sync(0xffffffffu, !kept)) {  // more than shared memory holds: walked again
        q0 = kept ? q0 : 0;
        rank = kept ? rank : 0;
        res_walk(a, r, s, s < n && !kept, skin, range, [&](bool hit, int e, bool) { enter(hit, e); });
      }
      __syncwarp();
    }
    if (!meet()) return;
    const unsigned long long ne = *(volatile unsigned long long*)r.total, np = *(volatile unsigned long long*)(r.total + 1);
    if (ne <= (unsigned long long)r.ent_cap && np <= (unsigned long long)r.pair_cap) break;
    if (skin == 0.) {  // more contacts than the lists hold
      if (tid == 0) {
        set_status(a.stats, GRAINS_GPU_PAIR_OVERFLOW);
        r.ctl[kResFailed] = 1;
      }
      return;
    }
    if (!meet()) return;  // every block has read the totals
    if (tid == 0) r.total[0] = r.total[1] = 0;
    if (!meet()) return;
    skin = skin < 1.e-3 * r.skin0 ? 0. : 0.5 * skin;  // without a skin: the contacts alone, built in every step
  }
  // each pair's entry in the partner's list, and its memory from the owner's row
  for (int s = group; s < padded; s += groups) {
    int2 en = make_int2(0, 0);
    int row = 0, hn = 0;
    if (s < n) {
      en = r.ent[s];
      row = a.cur.orig[s];
      hn = a.hist_n_prev[row];
    }
    const HistEntry<R>* h = a.hist_prev + (size_t)row * a.hist_cap;
    for (int q = lane; q < en.y; q += kResLanes) {
      const int e = r.nb[en.x + q];
      if (!(e & kOwnBit)) continue;
      const int mine = r.ent_pair[en.x + q];
      const int t = entry_slot(e);
      const int2 te = r.ent[t];
      const int id = a.cur.meta[t].x;
      int other = -1;
      for (int k = 0; k < te.y; ++k)
        if (r.nb[te.x + k] == s) other = te.x + k;
      r.pair[mine].w = other;
      if (other >= 0) r.ent_pair[other] = mine;
      if (r.konst) r.konst[mine] = res_constants(a, s, t);
      unsigned char st = 0;
      for (int k = 0; k < hn; ++k)
        if (h[k].other == id && h[k].flags == 0) {
          PairMemory<R> m;
          m.kdelta = v3<R>(h[k].kd[0], h[k].kd[1], h[k].kd[2]);
          m.prev_normal = v3<R>(h[k].n[0], h[k].n[1], h[k].n[2]);
          m.spring = v3<R>(h[k].sp[0], h[k].sp[1], h[k].sp[2]);
          res_store_memory(r.mem + mine, (size_t)r.pair_cap, m, true);
          st = kResContact | kResMemory;
          break;
        }
      r.state[mine] = st;
    }
  }
  if (!meet()) return;
  if (tid == 0) {
    *r.skin = skin;
    r.ctl[kResValid] = (int)r.total[1];
    r.ctl[kResRowPairs] = 0;
    r.ctl[kResRequest] = 0;
  }
}

// ---- obstacles ------------------------------------------------------------------
// The obstacles linked to the particle's cell whose box meets its sphere's box
// (the candidates of contacts_one): bit o for the system's obstacle o.
template <typename R>
__device__ __forceinline__ unsigned res_obstacle_candidates(const StepArgs<R>& a, const SysDev& S, unsigned key, D3 X,
                                                            double radius) {
  unsigned mask = 0;
  const int b = a.cell_obs_start[key], e = a.cell_obs_start[key + 1];
  for (int u = b; u < e; ++u) {
    const int o = a.cell_obs_idx[u];
    const ObstacleDev& O = a.obs[o];
    if (in_zone(d3(O.bbc[0], O.bbc[1], O.bbc[2]), d3(O.bbe[0], O.bbe[1], O.bbe[2]), X, radius, radius, radius))
      mask |= 1u << (o - S.obs_offset);
  }
  return mask;
}

// candidates `mask` of particle s (every lane of the warp calls it, a lane
// without a particle with an empty mask): items for the evaluation of parity
// `parity`; returns the state word, in which obstacles that are no candidates
// have lost their contact
template <typename R>
__device__ __forceinline__ unsigned long long res_emit_obstacles(const ResArgs<R>& r, int s, unsigned mask,
                                                                 unsigned long long state, int parity) {
  const int base = warp_reserve(r.ctl + kResObs + parity, __popc(mask));
  unsigned long long next = 0;
  int k = base;
  for (unsigned m = mask; m; m &= m - 1) {
    const int o = __ffs(m) - 1;
    next |= (((state >> (8 * o)) & (kResContact | kResMemory)) | kResCandidate) << (8 * o);
    r.obs_item[parity][k++] = s * kResObsMax + o;
  }
  return next;
}

// the start of a run: the obstacle candidates of the current positions and
// their memory from the rows
template <typename R>
__global__ void __launch_bounds__(256) res_begin_kernel(StepArgs<R> a, ResArgs<R> r) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  const bool active = s < a.n;
  unsigned mask = 0;
  unsigned long long state = 0;
  if (active) {
    const double4 x = a.cur.xr[s];
    const SysDev& S = a.sys[a.cur.meta[s].w];
    mask = res_obstacle_candidates(a, S, a.cur.key[s], d3(x.x, x.y, x.z), x.w);
    const int row = a.cur.orig[s];
    const HistEntry<R>* h = a.hist_prev + (size_t)row * a.hist_cap;
    for (int k = a.hist_n_prev[row] - 1; k >= 0; --k) {  // the first of equal entries counts
      const int o = h[k].other;
      if (h[k].flags != 1 || o < 0 || o >= S.n_obs || !((mask >> o) & 1)) continue;
      PairMemory<R> m;
      m.kdelta = v3<R>(h[k].kd[0], h[k].kd[1], h[k].kd[2]);
      m.prev_normal = v3<R>(h[k].n[0], h[k].n[1], h[k].n[2]);
      m.spring = v3<R>(h[k].sp[0], h[k].sp[1], h[k].sp[2]);
      res_store_memory(r.obs_mem + 9 * ((size_t)s * r.obs_stride + o), 1, m, true);
      state |= (unsigned long long)(kResContact | kResMemory) << (8 * o);
    }
  }
  const unsigned long long next = res_emit_obstacles(r, s, mask, state, 0);
  if (active) r.obs_state[s] = next;
  if (s == 0) {
    r.ctl[kResRequest] = 2;
    r.ctl[kResValid] = -1;
    r.ctl[kResCountAll] = 1;
  }
}

// the end of a run: every memory back into the rows, pairs then obstacles.  Without
// complete lists the rows hold everything (a first build), or the pairs' memories
// (a rebuild that failed)
template <typename R>
__global__ void __launch_bounds__(256) res_end_kernel(StepArgs<R> a, ResArgs<R> r) {
  const bool valid = *(volatile int*)(r.ctl + kResValid) >= 0;
  if (!valid && !*(volatile int*)(r.ctl + kResRowPairs)) return;
  const int s = (blockIdx.x * blockDim.x + threadIdx.x) / kResLanes;
  const bool active = s < a.n;
  int cnt = valid ? res_flush_pairs(a, r, s, active) : 0;
  if (!active || res_lane() != 0) return;
  const unsigned long long state = r.obs_state[s];
  if (!state) return;
  const int row = a.cur.orig[s];
  if (!valid) cnt = a.hist_n_prev[row];
  HistEntry<R>* h = a.hist_prev + (size_t)row * a.hist_cap;
  for (int o = 0; o < kResObsMax; ++o) {
    if (!((state >> (8 * o)) & kResMemory)) continue;
    const PairMemory<R> m = res_load_memory(r.obs_mem + 9 * ((size_t)s * r.obs_stride + o), 1, true);
    if (cnt >= a.hist_cap) {
      set_status(a.stats, GRAINS_GPU_HISTORY_FULL);
      break;
    }
    HistEntry<R> x;
    x.other = o;
    x.flags = 1;
    x.kd[0] = m.kdelta.x; x.kd[1] = m.kdelta.y; x.kd[2] = m.kdelta.z;
    x.n[0] = m.prev_normal.x; x.n[1] = m.prev_normal.y; x.n[2] = m.prev_normal.z;
    x.sp[0] = m.spring.x; x.sp[1] = m.spring.y; x.sp[2] = m.spring.z;
    h[cnt++] = x;
  }
  a.hist_n_prev[row] = cnt;
}

// ---- pairs ----------------------------------------------------------------------
constexpr int kResPairThreads = 128;

template <typename R>
__device__ __forceinline__ void res_no_contact(const ResArgs<R>& r, int p, int4 pr) {
  if (!r.state[p]) return;
  r.state[p] = 0;
  r.res[pr.z].f.w = R(0);
  if (pr.w >= 0) r.res[pr.w].f.w = R(0);
}

// the results, memory and state of listed pair p after its law
template <typename R>
__device__ __forceinline__ void res_put_pair(const ResArgs<R>& r, int p, int4 pr, unsigned char st, bool memory,
                                             const ContactGeom& g, V3<R> f, V3<R> t0, V3<R> t1, ForceStats& fs) {
  const int now = memory ? kResContact | kResMemory : kResContact;
  if (st != now) r.state[p] = (unsigned char)now;
  r.res[pr.z].f = st3<R>(f, R(memory ? 3 : 2));
  r.res[pr.z].t = st3<R>(t0);
  if (pr.w >= 0) {
    r.res[pr.w].f = st3<R>(-f, R(1));
    r.res[pr.w].t = st3<R>(t1);
  }
  ++fs.ncont_own;
  const double o = fabs(g.overlap);
  fs.ov_sum += o;
  fs.ov_max = fmax(fs.ov_max, o);
}

// the contact law of listed pair p (in contact: the overlap test has passed)
template <typename R>
__device__ __forceinline__ void res_pair_any_law(const StepArgs<R>& a, const ResArgs<R>& r, int p, R dt,
                                                 ForceStats& fs) {
  const ParticleArrays<R>& P = a.cur;
  const int4 pr = r.pair[p];
  const int s = pr.x, t = pr.y;
  const double4 xi = P.xr[s], xj = P.xr[t];
  const int4 mi = P.meta[s], mj = P.meta[t];
  const double4 mdi = P.md[s], mdj = P.md[t];
  const V3<R> vi = ld3<R>(P.v[s]), wi = ld3<R>(P.w[s]);
  const V3<R> vj = ld3<R>(P.v[t]), wj = ld3<R>(P.w[t]);
  const unsigned char st = r.state[p];
  const SysDev& S = a.sys[mi.w];
  const LawParams<R> L = a.laws[S.law_offset + mi.y * S.n_mat + mj.y];
  const bool memory = law_has_memory(L.type);
  PairMemory<R> mem;
  const bool existed = memory && (st & kResMemory);
  if (existed) mem = res_load_memory(r.mem + p, (size_t)r.pair_cap, L.rolling != 0);
  const D3 Xi = d3(xi.x, xi.y, xi.z), Xj = d3(xj.x, xj.y, xj.z);
  ContactGeom g;
  if (!sphere_pair_geometry(a, Xi, xi.w, mdi.y, Xj, xj.w, mdj.y, g)) {
    res_no_contact(r, p, pr);
    return;
  }
  V3<R> t0, t1;
  const LawResult<R> res = particle_pair_law(L, dt, g, Xi, Xj, mdi, mdj, vi, wi, vj, wj, existed, mem, t0, t1);
  if (memory) res_store_memory(r.mem + p, (size_t)r.pair_cap, mem, L.rolling != 0 || !existed);
  if (law_has_torque(L)) {
    t0 = t0 + res.torque;
    t1 = t1 + (-res.torque);
  }
  res_put_pair(r, p, pr, st, memory, g, res.force, t0, t1, fs);
}

// The same for a context whose only law is HookeMemory without a rolling spring:
// what depends on the two bodies alone (the damping coefficients, the crust sum,
// the law's slot) comes from the pair's constants, formed by the build with the
// law's own expressions.  That leaves out the gathers of both bodies' masses and
// materials, and four divisions and two square roots of the chain.
template <typename R>
__device__ __forceinline__ void res_pair_hooke_memory(const StepArgs<R>& a, const ResArgs<R>& r, int p, R dt,
                                                      ForceStats& fs) {
  const ParticleArrays<R>& P = a.cur;
  const int4 pr = r.pair[p];
  const ResConst k = r.konst[p];
  const unsigned char st = r.state[p];
  const int s = pr.x, t = pr.y;
  const double4 xi = P.xr[s], xj = P.xr[t];
  BodyAtContact<R> b0, b1;
  b0.v = ld3<R>(P.v[s]);
  b0.w = ld3<R>(P.w[s]);
  b1.v = ld3<R>(P.v[t]);
  b1.w = ld3<R>(P.w[t]);
  const LawParams<R>& L = a.laws[k.law];
  const bool existed = (st & kResMemory) != 0;
  PairMemory<R> mem;
  if (existed) mem = res_load_memory(r.mem + p, (size_t)r.pair_cap, false);
  const D3 Xi = d3(xi.x, xi.y, xi.z), Xj = d3(xj.x, xj.y, xj.z);
  D3 ab;
  double nab;
  const double dist = sphere_sphere_overlap(Xi, xi.w, Xj, xj.w, &ab, &nab);
  ContactGeom g = sphere_sphere_features(Xi, xi.w, ab, nab, dist, k.crust);
  if (g.status && !sphere_pair_geometry(a, Xi, xi.w, P.md[s].y, Xj, xj.w, P.md[t].y, g)) {
    res_no_contact(r, p, pr);
    return;
  }
  const D3 lev0 = xsub3(g.point, Xi), lev1 = xsub3(g.point, Xj);
  b0.lever = from_d3<R>(lev0);
  b1.lever = from_d3<R>(lev1);
  V3<R> f, t0, t1;
  if constexpr (sizeof(R) == 4) {
    // normal_part_fp64 and pair_law, with the constants
    const V3<double> pen = v3<double>(g.overlap_vector.x, g.overlap_vector.y, g.overlap_vector.z);
    const V3<double> l0 = dvec(lev0), l1 = dvec(lev1);
    const V3<double> normal = round3(dv(pen, norm(pen)));
    const V3<double> rel = (widen(b0.v) + cross(widen(b0.w), l0)) - (widen(b1.v) + cross(widen(b1.w), l1));
    const V3<double> v_n = sc(normal, dot(rel, normal));
    const V3<double> v_t = rel - v_n;
    const V3<double> fn = sc(pen, L.kn64) - sc(v_n, k.gamman);
    const LawResult<R> res = memory_tangent_rolling(
        L, dt, v3<R>(R(normal.x), R(normal.y), R(normal.z)), v3<R>(R(v_t.x), R(v_t.y), R(v_t.z)),
        v3<R>(R(fn.x), R(fn.y), R(fn.z)), R(norm(fn)), R(k.gammat), L.kt, R(L.kn64), R(k.gamman), b0, b1, existed, mem,
        (int*)nullptr, false);
    const V3<double> tn0 = cross(l0, fn), tn1 = cross(l1, -fn);
    f = res.force;
    t0 = v3<R>(R(tn0.x), R(tn0.y), R(tn0.z)) + cross(b0.lever, res.tangential);
    t1 = v3<R>(R(tn1.x), R(tn1.y), R(tn1.z)) + cross(b1.lever, -res.tangential);
  } else {
    // hooke_memory, with the constants
    const V3<R> pen = from_d3<R>(g.overlap_vector);
    const V3<R> normal = round3(dv(pen, norm(pen)));
    const V3<R> rel = velocity_at(b0) - velocity_at(b1);
    const V3<R> v_n = sc(normal, dot(rel, normal));
    const V3<R> v_t = rel - v_n;
    const V3<R> fn = sc(pen, L.kn) - sc(v_n, R(k.gamman));
    const LawResult<R> res = memory_tangent_rolling(L, dt, normal, v_t, fn, norm(fn), R(k.gammat), L.kt, L.kn,
                                                    R(k.gamman), b0, b1, existed, mem, (int*)nullptr, false);
    f = res.force;
    t0 = cross(b0.lever, res.force);
    t1 = cross(b1.lever, -res.force);
  }
  res_store_memory(r.mem + p, (size_t)r.pair_cap, mem, !existed);
  res_put_pair(r, p, pr, st, true, g, f, t0, t1, fs);
}

// one obstacle candidate (pair_one's obstacle part on resident memory)
template <typename R>
__device__ __forceinline__ void res_obstacle_one(const StepArgs<R>& a, const ResArgs<R>& r, int item, R dt,
                                                 ForceStats& fs) {
  const ParticleArrays<R>& P = a.cur;
  const int s = item / kResObsMax, o = item % kResObsMax;
  const double4 xi = P.xr[s];
  const int4 mi = P.meta[s];
  const double4 mdi = P.md[s];
  const V3<R> vi = ld3<R>(P.v[s]), wi = ld3<R>(P.w[s]);
  unsigned char* state = reinterpret_cast<unsigned char*>(r.obs_state + s) + o;
  const unsigned char st = *state;
  const SysDev& S = a.sys[mi.w];
  const ObstacleDev& O = a.obs[S.obs_offset + o];
  const size_t at = (size_t)s * r.obs_stride + o;
  const D3 Xi = d3(xi.x, xi.y, xi.z);
  const ShapeDev& sho = a.shapes[O.shape];
  M3 ob;
  for (int k = 0; k < 9; ++k) ob.m[k] = O.b[k];
  ContactGeom g = sphere_box(Xi, xi.w, xadd(mdi.y, O.crust), ob, d3(O.o[0], O.o[1], O.o[2]),
                             d3(sho.ext[0], sho.ext[1], sho.ext[2]));
  if (g.status) {
    set_status(a.stats, GRAINS_GPU_CONTACT_ERROR);
    g.overlap = 1.;
  }
  if (!(g.overlap < 0.)) {
    if (st != kResCandidate) *state = kResCandidate;
    return;
  }
  const LawParams<R> L = a.laws[S.law_offset + mi.y * S.n_mat + O.material];
  const bool memory = law_has_memory(L.type);
  PairMemory<R> mem;
  const bool existed = memory && (st & kResMemory);
  if (existed) mem = res_load_memory(r.obs_mem + 9 * at, 1, L.rolling != 0);
  V3<R> t0, t1;
  const LawResult<R> res = obstacle_law(L, dt, g, Xi, O, sho, mdi, vi, wi, existed, mem, t0, t1);
  if (memory) res_store_memory(r.obs_mem + 9 * at, 1, mem, L.rolling != 0 || !existed);
  const int now = kResCandidate | kResContact | (memory ? kResMemory : 0);
  if (st != now) *state = (unsigned char)now;
  if (law_has_torque(L)) t0 = t0 + res.torque;
  r.obs_res[at].f = st3<R>(res.force, R(memory ? 3 : 1));
  r.obs_res[at].t = st3<R>(t0);
  ++fs.nobs_cont;
  const double ov = fabs(g.overlap);
  fs.ov_sum += ov;
  fs.ov_max = fmax(fs.ov_max, ov);
}

// The number of candidate pairs of the step (the 27 cells around every particle,
// as the launched broadphase counts them), and the cell counts of the next step
// cleared.  With n the cells' counts and A their adjacency (27 cells), the number
// is n.An - N; a step changes few cells, and with d = n_new - n_old the change is
// d.(A n_old + A n_new), so only cells whose count has changed look around.
// Counting all cells took 20 us of a step of 200,000 falling spheres and 140 us of
// one of 500 systems (5 million cells).  The sums kernel adds the number to the
// statistics.
template <typename R>
__device__ __forceinline__ void res_count_candidates(const StepArgs<R>& a, const ResArgs<R>& r, int step, int block,
                                                     int blocks) {
  const int* now = r.count[step % 3];
  const int* old = r.count[(step + 2) % 3];
  int* next = r.count[(step + 1) % 3];
  const bool all = *(volatile int*)(r.ctl + kResCountAll) != 0;
  long long sum = 0;
  auto around = [&](int c) {  // the 27 cells of c: of both counts (of the new one alone when all cells are counted)
    int sys = 0;
    for (int hi = a.n_sys; hi - sys > 1;) {  // the cell's system
      const int mid = (sys + hi) / 2;
      if (a.sys[mid].cell_offset <= c) sys = mid;
      else hi = mid;
    }
    const SysDev& S = a.sys[sys];
    const int local = c - S.cell_offset;
    const int i = local % S.nbi, k = (local / S.nbi) % S.nbk, j = local / (S.nbi * S.nbk);
    int m = 0;
#pragma unroll 9
    for (int q = 0; q < 27; ++q) {
      const int ii = i + q % 3 - 1, kk = k + (q / 3) % 3 - 1, jj = j + q / 9 - 1;
      if (ii >= 0 && ii < S.nbi && jj >= 0 && jj < S.nbj && kk >= 0 && kk < S.nbk) {
        const int o = cell_index(S, ii, jj, kk);
        m += now[o];
        if (!all) m += old[o];
      }
    }
    return m;
  };
  const int quads = (a.n_cells + 3) / 4;
  for (int q = block * kResPairThreads + threadIdx.x; q < quads; q += blocks * kResPairThreads) {
    const int c = 4 * q;
    int n4[4], o4[4];
    if (c + 4 <= a.n_cells) {
      const int4 x = reinterpret_cast<const int4*>(now)[q], y = reinterpret_cast<const int4*>(old)[q];
      reinterpret_cast<int4*>(next)[q] = make_int4(0, 0, 0, 0);
      n4[0] = x.x; n4[1] = x.y; n4[2] = x.z; n4[3] = x.w;
      o4[0] = y.x; o4[1] = y.y; o4[2] = y.z; o4[3] = y.w;
    } else {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const bool in = c + u < a.n_cells;
        n4[u] = in ? now[c + u] : 0;
        o4[u] = in ? old[c + u] : 0;
        if (in) next[c + u] = 0;
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int d = all ? n4[u] : n4[u] - o4[u];
      if (d != 0) sum += (long long)d * around(c + u);
    }
  }
  warp_add(r.n_cand, (unsigned long long)sum);  // two's complement: changes may be negative
}

// Blocks [0, pair_blocks): the listed pairs.  Each warp tests 32 or 64 pairs at a
// time (the exact overlap test of every listed pair) and queues those in contact
// in shared memory; whenever 32 are queued it runs the law on them, so that the
// law runs on full warps whatever share of the list is in contact, without a
// barrier.  64 at a time keeps twice the loads in flight; 32 spreads a short list
// over more warps.  Then obs_blocks: the obstacle candidates; the other blocks:
// res_count_candidates.
// Bound by the latency of the gathers and by L2 (390 B a contact); four
// blocks a SM at 128 registers (five at 96 spill: 67.2 against 66.5 us).  200,000
// spheres, 460,000 contacts: 82 -> 66 us mixed, 103 -> 82 us FP64 with the pair
// constants and without the block-wide barriers of the first form.
constexpr int kResPairBlocks = 4;
template <typename R, bool HOOKE_MEMORY>
__global__ void __launch_bounds__(kResPairThreads, kResPairBlocks)
    res_pairs_kernel(StepArgs<R> a, ResArgs<R> r, R dt, int step, int pair_blocks, int obs_blocks) {
  const int parity = step & 1;
  constexpr int kQueue = 96;
  __shared__ int queue_s[kResPairThreads / 32][kQueue];
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  ForceStats fs{0, 0, 0, 0, 0., 0.};
  if ((int)blockIdx.x < pair_blocks) {
    const int n_pairs = *(volatile int*)(r.ctl + kResValid);
    int* queue = queue_s[threadIdx.x / 32];
    const int warps = pair_blocks * (kResPairThreads / 32);
    const int warp = blockIdx.x * (kResPairThreads / 32) + threadIdx.x / 32;
    const int per = n_pairs > 32 * warps ? 2 : 1;
    int queued = 0;
    auto law = [&](int p) {
      if constexpr (HOOKE_MEMORY)
        res_pair_hooke_memory(a, r, p, dt, fs);
      else
        res_pair_any_law(a, r, p, dt, fs);
    };
    bool more = true;
    for (int base = warp * 32 * per; more; base += warps * 32 * per) {
      more = base < n_pairs;
      if (more) {
        int4 pr[2];
        double4 xi[2], xj[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int p = base + 32 * u + lane;
          pr[u] = u < per && p < n_pairs ? r.pair[p] : make_int4(0, 0, 0, 0);
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          xi[u] = a.cur.xr[pr[u].x];
          xj[u] = a.cur.xr[pr[u].y];
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int p = base + 32 * u + lane;
          bool contact = false;
          if (u < per && p < n_pairs) {
            const double dx = xj[u].x - xi[u].x, dy = xj[u].y - xi[u].y, dz = xj[u].z - xi[u].z;
            const double rs = xi[u].w + xj[u].w;
            if (!(dx * dx + dy * dy + dz * dz > rs * rs * (1. + 1.e-12))) {  // as the broadphase tests
              D3 ab;
              double nab;
              contact = sphere_sphere_overlap(d3(xi[u].x, xi[u].y, xi[u].z), xi[u].w,
                                              d3(xj[u].x, xj[u].y, xj[u].z), xj[u].w, &ab, &nab) < 0.;
            }
            if (!contact) res_no_contact(r, p, pr[u]);
          }
          const unsigned hit = __ballot_sync(full, contact);
          if (contact) queue[queued + __popc(hit & ((1u << lane) - 1u))] = p;
          queued += __popc(hit);
        }
        __syncwarp();
      }
      // full warps as they come, the rest in the end
      while (queued >= 32 || (!more && queued > 0)) {
        const int take = min(queued, 32);
        const int p = lane < take ? queue[queued - take + lane] : -1;
        queued -= take;
        __syncwarp();
        if (p >= 0) law(p);
        __syncwarp();
      }
    }
    flush_force_stats(a.stats, fs);
  } else if ((int)blockIdx.x < pair_blocks + obs_blocks) {
    // (no lists: the run stands still, its obstacles too)
    const int valid = *(volatile int*)(r.ctl + kResValid), listed = *(volatile int*)(r.ctl + kResObs + parity);
    const int n_items = valid >= 0 ? listed : 0;
    const int b = blockIdx.x - pair_blocks;
    for (int k = b * kResPairThreads + threadIdx.x; k < n_items; k += obs_blocks * kResPairThreads)
      res_obstacle_one(a, r, r.obs_item[parity][k], dt, fs);
    if (b == 0 && threadIdx.x == 0) {
      if (n_items > 0) atomicAdd(&a.stats->n_obs_cand, (unsigned long long)n_items);
      r.ctl[kResObs + 1 - parity] = 0;  // the sums kernel fills the next step's list
    }
    flush_force_stats(a.stats, fs);
  } else {
    res_count_candidates(a, r, step, blockIdx.x - pair_blocks - obs_blocks, gridDim.x - pair_blocks - obs_blocks);
  }
}

// ---- sums -----------------------------------------------------------------------

// The list of particle s back into the order of (cell, id) after partners have
// crossed into other cells: an insertion sort of the nearly ordered entries with
// their results; each moved entry's pair learns the new place.
template <typename R>
__device__ __forceinline__ void res_reorder(const StepArgs<R>& a, const ResArgs<R>& r, int2 en) {
  auto rank = [&](int e) {
    const int t = entry_slot(e);
    return ((unsigned long long)a.cur.key[t] << 32) | ((unsigned)a.cur.meta[t].x ^ 0x80000000u);
  };
  auto place = [&](int q, int e, int p, const ResResult<R>& x) {
    r.nb[q] = e;
    r.ent_pair[q] = p;
    r.res[q] = x;
    if (e & kOwnBit)
      r.pair[p].z = q;
    else
      r.pair[p].w = q;
  };
  unsigned long long last = 0;
  for (int q = en.x; q < en.x + en.y; ++q) {
    const int e = r.nb[q];
    const unsigned long long k = rank(e);
    if (q == en.x || k > last) {
      last = k;
      continue;
    }
    const int p = r.ent_pair[q];
    const ResResult<R> x = r.res[q];
    int to = q;
    for (; to > en.x; --to) {
      const int f = r.nb[to - 1];
      if (rank(f) < k) break;
      place(to, f, r.ent_pair[to - 1], r.res[to - 1]);
    }
    place(to, e, p, x);
  }
}

// `integrate` for a sphere whose torsor (F, T) is final: the second half kick,
// the next first half kick, the drift and the cell of the new position.  The same
// operations; what both kicks share is formed once, since the angular
// acceleration of a sphere does not depend on its rate (its three Runge-Kutta
// stages are equal), and divisions, the square root of the motion test and the
// cell's divisions take cheaper forms with the same results.  1,876 instructions
// a warp before.  B200, sums of 200,000 spheres: falling 25.3 -> 18.2 us, in a bed
// 44.6 -> 40.5 us mixed and 72.5 -> 60.4 us FP64.
template <typename R>
__device__ __forceinline__ void res_drift(const StepArgs<R>& a, const SysDev& S, const ParticleArrays<R>& P,
                                          unsigned* key_out, int s, const double4& md, V3<R> F, V3<R> T, R dt_half,
                                          double dt, D3& X, unsigned& key) {
  double4 xr = P.xr[s];
  const double4 qd = P.q[s];
  V3<R> v = ld3<R>(P.v[s]), w, wbf = ld3<R>(P.wbf[s]);
  const V3<R> I = ld3<R>(P.inertia[s]);
  const R mass = R(md.x);
  const R cf = a.fluid_corrected ? R(1. - md.w) : R(1);
  Qt<double> q{v3<double>(qd.x, qd.y, qd.z), qd.w};
  const Qt<R> qr{v3<R>(R(qd.x), R(qd.y), R(qd.z)), R(qd.w)};
  const V3<R> Tbf = q_to_body(qr, T);
  const V3<R> dvel = sc(div3(F, mass * cf), dt_half);
  const V3<R> at = v3<R>(Divisor<R>(cf * I.x)(Tbf.x), Divisor<R>(cf * I.y)(Tbf.y), Divisor<R>(cf * I.z)(Tbf.z));
  const V3<R> K = sc(at, dt_half);
  const V3<R> dw = div3((K + K) + sc(K, R(4)), R(6));  // rk3
  v = v + dvel;
  v = v + dvel;
  wbf = wbf + dw;
  wbf = wbf + dw;
  w = q_to_world(qr, wbf);
  const V3<double> tm = sc(v3<double>(double(v.x), double(v.y), double(v.z)), dt);
  xr.x = xr.x + tm.x;
  xr.y = xr.y + tm.y;
  xr.z = xr.z + tm.z;
  const V3<double> mw = v3<double>(double(w.x), double(w.y), double(w.z));
  const double nom = norm(mw);
  Qt<double> dq{v3<double>(0., 0., 0.), 1.};
  if (nom > kEpsilon) {
    const double c = cos(nom * dt / 2.), sn = sin(nom * dt / 2.);
    dq = Qt<double>{sc(mw, sn * 1. / nom), c};
  }
  q = qmul(dq, q);
  if (a.has_basis) {
    M3 b;
    for (int t = 0; t < 9; ++t) b.m[t] = P.basis[9 * (size_t)s + t];
    mrotate_left(b, dq);
    for (int t = 0; t < 9; ++t) P.basis[9 * (size_t)s + t] = b.m[t];
  }
  if (longer(tm, md.y)) set_status(a.stats, GRAINS_GPU_MOTION_ERROR);
  int ci, cj, ck;
  if (!cell_of(S, xr.x, xr.y, xr.z, ci, cj, ck)) set_status(a.stats, GRAINS_GPU_OUT_OF_GRID);
  key = (unsigned)cell_index(S, ci, cj, ck);
  key_out[s] = key;
  atomicAdd(&a.cell_count[key], 1);
  P.xr[s] = xr;
  P.q[s] = make_double4(q.v.x, q.v.y, q.v.z, q.w);
  P.v[s] = st3<R>(v);
  P.w[s] = st3<R>(w);
  P.wbf[s] = st3<R>(wbf);
  X = d3(xr.x, xr.y, xr.z);
}

// The torsor of particle s from the results of its list entries in the order of
// (cell of the partner, id), as the launched pipeline lists them; then its
// obstacles, the fluid, the kicks, the drift and the next step's candidates.
// Lists keep that order from their build; a particle that crosses into another
// cell marks its partners' lists for res_reorder in the next step (about one
// list in a hundred a step), so that no step looks up the partners' cells.
template <typename R>
__global__ void __launch_bounds__(256, 3) res_sums_kernel(StepArgs<R> a, ResArgs<R> r, R dt_half, double dt, int step) {
  const int parity = step & 1;
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  const bool valid = *(volatile int*)(r.ctl + kResValid) >= 0, active = s < a.n && valid;
  const ParticleArrays<R>& P = a.cur;
  if (s == 0) {
    if (valid) a.stats->n_cand += *r.n_cand - (unsigned long long)a.n;  // less the particles themselves
    r.ctl[kResCountAll] = 0;
  }
  if (s < a.n && !valid) {  // the particle stays; its key and count go on to the next step's arrays
    const unsigned key = P.key[s];
    a.alt.key[s] = key;
    atomicAdd(&a.cell_count[key], 1);
  }
  unsigned mask = 0;
  unsigned long long state = 0;
  if (active) {
    const int2 en = r.ent[s];
    const unsigned char dirty = r.dirty[parity][s];
    const int4 meta = P.meta[s];
    const double4 md = P.md[s];
    const unsigned old_key = P.key[s];
    state = r.obs_state[s];
    const double mass = md.x * (1. - md.w);  // Particle::computeWeight, as in sum_one
    const SysDev& S = a.sys[meta.w];
    V3<R> F = v3<R>(R(S.gx * mass), R(S.gy * mass), R(S.gz * mass));
    V3<R> T = v3<R>(R(0), R(0), R(0));
    if (dirty) {
      res_reorder(a, r, en);
      r.dirty[parity][s] = 0;
    }
    int listed = 0, owned = 0;
    bool full = false;  // a memory beyond the row
    for (int q0 = 0; q0 < en.y; q0 += 4) {
      ResResult<R> x[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (q0 + u < en.y) x[u] = r.res[en.x + q0 + u];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (q0 + u >= en.y || x[u].f.w == R(0)) continue;
        F = F + ld3<R>(x[u].f);
        T = T + ld3<R>(x[u].t);
        ++listed;
        full = full || (x[u].f.w == R(3) && owned >= a.hist_cap);
        owned += x[u].f.w >= R(2) ? 1 : 0;
      }
    }
    int n_cand = 0;
    for (unsigned long long m = state; m; ) {
      const int o = (__ffsll((long long)m) - 1) / 8;
      const unsigned b = (unsigned)(m >> (8 * o)) & 255u;
      m &= ~(255ull << (8 * o));
      if (!(b & kResCandidate)) continue;
      ++n_cand;
      if (b & kResContact) {
        const ResResult<R> x = r.obs_res[(size_t)s * r.obs_stride + o];
        F = F + ld3<R>(x.f);
        T = T + ld3<R>(x.t);
        full = full || (x.f.w == R(3) && owned >= a.hist_cap);
      }
      ++owned;
    }
    if (listed + n_cand > a.clist_cap) set_status(a.stats, GRAINS_GPU_PAIR_OVERFLOW);
    if (full) set_status(a.stats, GRAINS_GPU_HISTORY_FULL);
    add_hydro(a, P.orig[s], F, T);
    D3 X;
    unsigned key;
    // partners still read this particle's present cell: the new one goes to the
    // other key array
    res_drift(a, S, P, a.alt.key, s, md, F, T, dt_half, dt, X, key);
    const double4 x0 = r.x0[s];
    const double dx = X.x - x0.x, dy = X.y - x0.y, dz = X.z - x0.z;
    const double half = *r.skin * (0.5 * (1. - 1.e-9));
    if (!(dx * dx + dy * dy + dz * dz < half * half)) r.ctl[kResRequest] = 1;
    if (key != old_key)
      for (int q = 0; q < en.y; ++q) r.dirty[1 - parity][entry_slot(r.nb[en.x + q])] = 1;
    mask = res_obstacle_candidates(a, S, key, X, x0.w);
  }
  const unsigned long long next = res_emit_obstacles(r, s, mask, state, 1 - parity);
  if (active && next != state) r.obs_state[s] = next;
}

// ---- launchers ------------------------------------------------------------------
template <typename R>
int res_rebuild_blocks(int n) {
  int dev = 0, sms = 0, per_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, res_rebuild_kernel<R>, 256, 0) != cudaSuccess ||
      per_sm < 1)
    return 0;
  const int need = grid_for((long long)kResLanes * n, 256);
  return std::max(1, std::min(std::min(per_sm, 4) * sms, need));
}

template <typename R>
int launch_res_begin(const StepArgs<R>& a, const ResArgs<R>& r, cudaStream_t s) {
  // control words, barrier, skin and candidate count lie side by side
  if (cudaMemsetAsync(r.ctl, 0, (char*)r.block_sums - (char*)r.ctl, s) != cudaSuccess) return GRAINS_GPU_CUDA_ERROR;
  res_begin_kernel<R><<<grid_for(a.n, 256), 256, 0, s>>>(a, r);
  return check_launch();
}

template <typename R>
int launch_res_end(const StepArgs<R>& a, const ResArgs<R>& r, cudaStream_t s) {
  res_end_kernel<R><<<grid_for((long long)kResLanes * a.n, 256), 256, 0, s>>>(a, r);
  return check_launch();
}

// phases (bits): 1 = rebuild when asked for, 2 = pairs, 4 = sums and kick.  The
// cell keys alternate between the two particle buffers: a.cur.key holds those of
// the step's positions, a.alt.key takes the next ones.
template <typename R>
int launch_res_step(const StepArgs<R>& args, const ResArgs<R>& r, cudaStream_t s, double dt, int step, int phases) {
  StepArgs<R> a = args;
  if (step & 1) std::swap(a.cur.key, a.alt.key);
  if (phases & 1) {
    StepArgs<R> a0 = a;
    ResArgs<R> r0 = r;
    void* kargs[] = {&a0, &r0, &step};
    if (cudaLaunchCooperativeKernel((const void*)res_rebuild_kernel<R>, dim3(r.rebuild_blocks), dim3(256), kargs, 0,
                                    s) != cudaSuccess)
      return GRAINS_GPU_CUDA_ERROR;
  }
  if (phases & 2) {
    // every SM filled once by the pair blocks, fewer when the lists (about 5 pairs a particle) are short; the
    // obstacle and count blocks follow them
    const int pb = std::min(kResPairBlocks * 148, grid_for(5ll * a.n, kResPairThreads));
    const int ob = std::min(148, grid_for(a.n, kResPairThreads));
    const int cb = std::min(2 * 148, grid_for(a.n_cells, 4 * kResPairThreads));
    if (r.konst)
      res_pairs_kernel<R, true><<<pb + ob + cb, kResPairThreads, 0, s>>>(a, r, R(dt), step, pb, ob);
    else
      res_pairs_kernel<R, false><<<pb + ob + cb, kResPairThreads, 0, s>>>(a, r, R(dt), step, pb, ob);
  }
  if (phases & 4) {
    StepArgs<R> an = a;
    an.cell_count = r.count[(step + 1) % 3];  // the drift counts the new cells for the next step
    // one warp a block while that spreads the particles over more SMs
    const int sb = a.n <= 32 * 148 ? 32 : (a.n <= 128 * 148 * 2 ? 64 : 256);
    res_sums_kernel<R><<<grid_for(a.n, sb), sb, 0, s>>>(an, r, R(0.5 * dt), dt, step);
  }
  return check_launch();
}
