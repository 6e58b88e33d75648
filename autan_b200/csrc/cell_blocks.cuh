// Blocks of consecutive owned cells with the data their neighbourhood needs laid out per block
// (included by euler_device.cu, inside its namespace).
//
// The gradient loop reads about 23 neighbour records a cell, but the cells of a compact block share
// them: a block of 32 cells of the hybrid channel in Morton order reads about 180 different records
// besides its own (64 cells 270). The block lists those once (GradBlocks::list) and each thread block
// copies them into shared memory in one round of independent loads; the stencil entries then name a
// record by its place there. What was a chain of dependent gathers through L1 and L2 (row, then record,
// chunk after chunk) becomes one gather per block and shared-memory reads.
//
// Stencil rows and limiter rows keep the sliced layout of the handle's own (32 cells a slice) with
// the record index replaced by the record's place in its block.
//
// The lists are built on the device, once per handle and block size, by sorting each block's
// candidates in shared memory (deterministic: the list is the sorted set).

template <class P>
struct GradBlocks {
  const int* off;              // per block, its first entry of list (n_blocks + 1)
  const int* list;             // record indices outside the block's own cells, ascending
  const typename P::C* st;     // {w, place} per stencil entry, at the positions of Dev::st
  const typename P::C* inc;    // {rel(x_f, x_c), other side's place}, at those of Dev::inc_rec
  const int* active;           // the blocks to launch over, or null: all
};

// Sorts key[0, count) ascending (count a power of two), every thread of the block taking part.
__device__ __forceinline__ void bitonic_sort(int* key, int count) {
  for (int k = 2; k <= count; k <<= 1) {
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int i = threadIdx.x; i < count / 2; i += blockDim.x) {
        const int lo = 2 * i - (i & (j - 1)), hi = lo + j;
        const bool up = (lo & k) == 0;
        const int x = key[lo], y = key[hi];
        if ((x > y) == up) {
          key[lo] = y;
          key[hi] = x;
        }
      }
      __syncthreads();
    }
  }
}

// The sorted set of key[0, count) (padded with INT_MAX to a power of two) into uniq; returns its
// size. part: blockDim.x + 1 ints of shared memory. Every thread of the block calls it.
__device__ __forceinline__ int sorted_set(int* key, int count, int* uniq, int* part) {
  int pow2 = 1;
  while (pow2 < count) pow2 <<= 1;
  for (int i = count + threadIdx.x; i < pow2; i += blockDim.x) key[i] = INT_MAX;
  __syncthreads();
  bitonic_sort(key, pow2);
  const int t = threadIdx.x, nt = blockDim.x;
  const int i0 = static_cast<int>(static_cast<long long>(count) * t / nt);
  const int i1 = static_cast<int>(static_cast<long long>(count) * (t + 1) / nt);
  int mine = 0;
  for (int i = i0; i < i1; ++i) mine += (i == 0 || key[i] != key[i - 1]) ? 1 : 0;
  part[t + 1] = mine;
  __syncthreads();
  if (t == 0) {
    part[0] = 0;
    for (int i = 0; i < nt; ++i) part[i + 1] += part[i];
  }
  __syncthreads();
  int at = part[t];
  for (int i = i0; i < i1; ++i)
    if (i == 0 || key[i] != key[i - 1]) uniq[at++] = key[i];
  const int total = part[nt];
  __syncthreads();
  return total;
}

// The place of x in the sorted set uniq[0, n) (x is in it).
__device__ __forceinline__ int place_of(const int* uniq, int n, int x) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int m = (lo + hi) >> 1;
    if (uniq[m] < x) lo = m + 1;
    else hi = m;
  }
  return lo;
}

// The records outside its own cells that block b's stencils and incidences read. FILL false: their
// number into counts[b]; else the list at off[b] and the block's pair rows. nb cells a block, the first
// nb threads one each; all kSortThreads sort (blocks of 32 cells sorted by 32 threads: 133 us where
// these take 52, 4 550-cell channel). Shared memory: 2 cap ints (cap: at least the block's entries
// and incidences).
constexpr int kSortThreads = 256;
template <class P, bool FILL>
__global__ void k_grad_blocks(Dev<P> d, int nb, int cap, int* counts, const int* off, int* list,
                              typename P::C* st, typename P::C* inc) {
  using C = typename P::C;
  extern __shared__ int block_keys[];
  __shared__ int part[kSortThreads + 1];
  __shared__ int n_keys;
  int* key = block_keys;
  int* uniq = block_keys + cap;
  const int c0 = blockIdx.x * nb, c1 = min(c0 + nb, d.n);
  const int c = static_cast<int>(threadIdx.x) < nb ? c0 + static_cast<int>(threadIdx.x) : d.n;
  if (threadIdx.x == 0) n_keys = 0;
  __syncthreads();
  auto each = [&](const int* start, const int* len, auto&& body) {
    if (c >= d.n) return;
    const long long base = start[c >> 5] + (c & 31);
    const int n = len[c];
    for (int j = 0; j < n; ++j) body(4 * (base + static_cast<long long>(j) * kSlice));
  };
  auto add = [&](const C* row) {
    const int x = index_of(row[3]);
    if (x < c0 || x >= c1) key[atomicAdd(&n_keys, 1)] = x;
  };
  each(d.st_start, d.st_len, [&](long long at) { add(d.st + at); });
  each(d.inc_start, d.inc_len, [&](long long at) { add(d.inc_rec + at); });
  __syncthreads();
  const int n = sorted_set(key, n_keys, uniq, part);
  if constexpr (!FILL) {
    if (threadIdx.x == 0) counts[blockIdx.x] = n;
  } else {
    for (int i = threadIdx.x; i < n; i += blockDim.x) list[off[blockIdx.x] + i] = uniq[i];
    auto fill = [&](const C* row, C* out) {
      const int x = index_of(row[3]);
      const int at = x >= c0 && x < c1 ? x - c0 : nb + place_of(uniq, n, x);
#pragma unroll
      for (int k = 0; k < 3; ++k) out[k] = row[k];
      out[3] = index_value<C>(at);
    };
    each(d.st_start, d.st_len, [&](long long at) { fill(d.st + at, st + at); });
    each(d.inc_start, d.inc_len, [&](long long at) { fill(d.inc_rec + at, inc + at); });
  }
}

// A row in shared memory.
__device__ __forceinline__ int read_row(const float* r, float* w) {
  const float4 v = *reinterpret_cast<const float4*>(r);
  w[0] = v.x, w[1] = v.y, w[2] = v.z;
  return __float_as_int(v.w);
}
__device__ __forceinline__ int read_row(const double* r, double* w) {
  const double2 u = *reinterpret_cast<const double2*>(r);
  const double2 v = *reinterpret_cast<const double2*>(r + 2);
  w[0] = u.x, w[1] = u.y, w[2] = v.x;
  return static_cast<int>(__double_as_longlong(v.y));
}
// The shared memory of a split gradient block: the rows of its cells' stencils and incidences, its
// records component by component, and (in the stencil rows' place, once they are read) the
// reconstruction words of its cells and the wave speeds of their faces.
struct GradShape {
  int st_rows, inc_rows;  // the most of a block
  int records;            // own cells and listed records of the largest block
  int faces;              // the most faces of a cell
};
constexpr int kStageW = 21;  // words per cell of the staged reconstruction record (odd: no conflicts)
template <class C>
__host__ __device__ __forceinline__ size_t grad_rows_bytes(const GradShape& s, int nb) {
  const size_t rows = static_cast<size_t>(s.st_rows) * 4 * sizeof(C);
  const size_t stage = static_cast<size_t>(nb) * (kStageW + s.faces) * sizeof(C);
  return ((rows > stage ? rows : stage) + 15) / 16 * 16;
}
template <class C>
__host__ __device__ __forceinline__ size_t grad_split_bytes(const GradShape& s, int nb) {
  return grad_rows_bytes<C>(s, nb) + static_cast<size_t>(s.inc_rows) * 4 * sizeof(C) +
         5 * static_cast<size_t>(s.records) * sizeof(C);
}
// Gradients, bounds, limiter and (DT) the CFL step as k_gradients, five threads per cell, one per
// component (the sums, bounds and limiter of a component need no other): the same operations in the
// same order on the same values. The block's rows arrive by TMA bulk copies (one thread, one mbarrier,
// bounded wait; they are static, so the copies start before the previous launch's end) while its
// threads gather the listed records, and from then on everything is read from shared memory. A thread
// per cell walks its entries in chunks of two to four dependent loads; here a mesh of a few thousand
// cells has five times the warps and three rounds of loads in all. It issues 1.8 times the
// instructions of k_gradients_occ7, so it is the form of meshes whose cells alone do not fill the
// chip: see choose_defaults for the line and the figures. Dynamic shared memory: grad_split_bytes.
constexpr int kSplit = 5;
constexpr int kSplitCells = 64;
template <class P, bool LIMIT, bool DT>
__global__ void __launch_bounds__(kSplit * kSplitCells, 4)
    k_gradients_split(Dev<P> d, GradBlocks<P> g, GradShape shape, double cfl, int local) {
  using C = typename P::C;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ __align__(8) unsigned long long bar;
  const int b = g.active != nullptr ? __ldg(g.active + blockIdx.x) : static_cast<int>(blockIdx.x);
  const int nt = blockDim.x, nb = nt / kSplit, t = threadIdx.x;
  const int k0 = t / nb, cell = t - k0 * nb;  // a warp's threads share their component
  const int c = b * nb + cell;
  const int s0 = b * (nb >> 5), s1 = min(s0 + (nb >> 5), d.n_slices);
  const int e0 = __ldg(d.st_start + s0), ne = __ldg(d.st_start + s1) - e0;
  const int i0 = __ldg(d.inc_start + s0), nf = __ldg(d.inc_start + s1) - i0;
  C* const st = reinterpret_cast<C*>(smem_raw);
  C* const fr = reinterpret_cast<C*>(smem_raw + grad_rows_bytes<C>(shape, nb));
  C* const rec = fr + 4 * shape.inc_rows;
  const int R = shape.records;
  const bool live = c < d.n && cell_active(d, c);
  const int len = live ? __ldg(d.st_len + c) : 0;
  const int il = live ? __ldg(d.inc_len + c) : 0;
  const C vol = live ? static_cast<C>(__ldg(d.volume + c)) : C(1);
  if (t == 0) {
    mbar_init(&bar, 1);
    const unsigned row = 4 * sizeof(C);
    const bool faces = (LIMIT || DT) && nf > 0;
    mbar_expect_tx(&bar, row * (static_cast<unsigned>(ne) + (faces ? static_cast<unsigned>(nf) : 0u)));
    if (ne > 0) bulk_to_shared(st, g.st + 4LL * e0, row * ne, &bar);
    if (faces) bulk_to_shared(fr, g.inc + 4LL * i0, row * nf, &bar);
  }
  dependents_may_start();
  previous_done();
  // the block's records: its own cells', then the listed ones'
  auto put = [&](int i, const C* w) {
#pragma unroll
    for (int k = 0; k < 5; ++k) rec[k * R + i] = w[k];
  };
  {
    const int n0 = __ldg(g.off + b), nu = __ldg(g.off + b + 1) - n0;
    const int own = min(nb, d.n - b * nb);
    for (int i = t; i < nb + nu; i += nt) {
      if (i >= nb || i < own) {
        const int x = i < nb ? b * nb + i : __ldg(g.list + n0 + i - nb);
        C u[5];
        load5<P, true>(d.prim + static_cast<long long>(x) * kPrimW, u);
        put(i, u);
      }
    }
  }
  __syncthreads();  // the records, and the barrier's initialisation
  const bool arrived = bounded_wait(&bar, d.ctl);
  if (__syncthreads_and(arrived ? 1 : 0) == 0) return;

  const int sl = (c >> 5) < s1 ? (c >> 5) : s0;
  const C* const row = st + 4 * (__ldg(d.st_start + sl) - e0 + (cell & 31));
  const C* const frow = fr + 4 * (__ldg(d.inc_start + sl) - i0 + (cell & 31));
  const C* const r0 = rec + k0 * R;
  const C wc = r0[cell];
  C lo = C(INFINITY), hi = -C(INFINITY);
  double acc[3] = {0.0, 0.0, 0.0};
#pragma unroll 4
  for (int j = 0; j < len; ++j) {
    C w[3];
    const C wn = r0[read_row(row + 4 * kSlice * j, w)];
    const C dw = wn - wc;
#pragma unroll
    for (int a = 0; a < 3; ++a) acc[a] += static_cast<double>(dw * w[a]);
    lo = bound_min(lo, wn);
    hi = bound_max(hi, wn);
  }
  C grad[3], phi = C(1.0);
#pragma unroll
  for (int a = 0; a < 3; ++a) grad[a] = static_cast<C>(acc[a]);
  if constexpr (LIMIT) {
    const C dmax = maxv(hi, wc) - wc, dmin = minv(lo, wc) - wc;
    const C eps2 = d.p.scale[k0] * vol;
    for (int j = 0; j < il; ++j) {
      C r[3];
      read_row(frow + 4 * kSlice * j, r);
      const C dd = grad[0] * r[0] + grad[1] * r[1] + grad[2] * r[2];
      phi = venkat_min(phi, dd, dmax, dmin, eps2);
    }
    phi = minv(phi, C(1.0));
  }
  __syncthreads();  // the stencil rows' place is free
  C* const stage = st;
  C* const speed = st + nb * kStageW;
  stage[cell * kStageW + k0] = phi;
#pragma unroll
  for (int a = 0; a < 3; ++a) stage[cell * kStageW + 5 + 3 * k0 + a] = grad[a];
  if constexpr (DT) {
    // the wave speeds of the cell's faces, shared out over its threads
    if (live) {
      C w[5];
#pragma unroll
      for (int k = 0; k < 5; ++k) w[k] = rec[k * R + cell];
      const C cc = sound_speed(w, d.p.g, d.p.pref);
      const long long ib = __ldg(d.inc_start + (c >> 5)) + (c & 31);
      for (int j = k0; j < il; j += kSplit) {
        C r[3];
        const int o = read_row(frow + 4 * kSlice * j, r);
        C nd[4], wn[5];
        load_words<P, sizeof(C) == 8>(d.inc_dt + 4 * (ib + static_cast<long long>(j) * kSlice), 0, 4, nd);
#pragma unroll
        for (int k = 0; k < 5; ++k) wn[k] = rec[k * R + o];
        speed[j * nb + cell] = wave_speed_cc(w, cc, wn, nd, nd[3], d.p.g, d.p.pref);
      }
    }
  }
  __syncthreads();
  for (int i = t; i < (kRecon / kGroup) * nb; i += nt) {
    const int gr = i / nb, cl = i - gr * nb;
    const int cc = b * nb + cl;
    if (cc < d.n && cell_active(d, cc)) {
      C o[kGroup];
#pragma unroll
      for (int e = 0; e < kGroup; ++e) o[e] = gr * kGroup + e < 20 ? stage[cl * kStageW + gr * kGroup + e] : C(0);
      store_words<P, true>(d.recon + gr * d.rstride + static_cast<long long>(cc) * kGroup, 0, kGroup, o);
    }
  }
  if constexpr (DT) {
    double dt = 0.0;
    if (live && k0 == 0) {
      double lam = 0.0;
      for (int j = 0; j < il; ++j) lam += static_cast<double>(speed[j * nb + cell]);
      dt = cfl * d.volume[c] / static_cast<double>(static_cast<C>(lam));
      if (local) d.dt_local[c] = dt;
    }
    block_min_dt(dt, live && k0 == 0, &d.ctl->dt_bits);
  }
}
