// The faces of blocks of consecutive owned cells (included by euler_device.cu, inside its namespace,
// after cell_blocks.cuh).

// A block's faces: every face that touches one of its cells, once, interior ones first, their records
// copied beside one another (kFace words, 16-byte piece q of face i of a block at rec[Q first + q n +
// i] with n its interior faces and Q pieces a record), then its boundary faces by index. A cell's
// incidences name them by their place, place * 2 + (1 if the flux is taken off), four 16-bit values to
// a load (sliced like the incidences, four to a row: row r of a cell at inc[start[slice] + 32 r + lane]).
// `walls` lists the boundary faces whose owner is in the block, the images' among them: their next
// boundary states follow from the owner's next primitives alone.
template <class P>
struct FaceBlocks {
  const int* first;    // per block, its first interior face record (n_blocks + 1)
  const int* bfirst;   // per block, its first entry of bface (n_blocks + 1)
  const typename P::V* rec;
  const int* face;     // the interior faces by index (the moments of warped faces)
  const int* bface;    // the boundary faces by index
  const uint2* inc;
  const int* inc_start;  // per slice
  const int* wfirst;   // per block, its first entry of walls (n_blocks + 1), or null: none are written
  const int* walls;
  const int* active;   // the blocks to launch over, or null: all
  int cells;           // cells per block
};

// The faces of block b: interior faces f as f, boundary faces b as n_if + b. FILL false: their numbers
// (interior, boundary) into counts[2 b], counts[2 b + 1]; else the block's lists, records and places.
// Threads as k_grad_blocks.
template <class P, bool FILL>
__global__ void k_face_blocks(Dev<P> d, int nb, int cap, int* counts, const int* first, const int* bfirst,
                              typename P::V* rec, int* face, int* bface, uint2* inc,
                              const int* inc_start) {
  using C = typename P::C;
  using V = typename P::V;
  extern __shared__ int block_keys[];
  __shared__ int part[kSortThreads + 1];
  __shared__ int n_keys, n_inner;
  int* key = block_keys;
  int* uniq = block_keys + cap;
  const int c = static_cast<int>(threadIdx.x) < nb ? static_cast<int>(blockIdx.x) * nb + static_cast<int>(threadIdx.x) : d.n;
  if (threadIdx.x == 0) n_keys = n_inner = 0;
  __syncthreads();
  const long long base = c < d.n ? d.inc_start[c >> 5] + (c & 31) : 0;
  const int il = c < d.n ? d.inc_len[c] : 0;
  auto key_of = [&](int code) { return code >= 0 ? code >> 1 : d.n_if + (-code - 1); };
  for (int j = 0; j < il; ++j)
    key[atomicAdd(&n_keys, 1)] = key_of(d.inc_code[base + static_cast<long long>(j) * kSlice]);
  __syncthreads();
  const int n = sorted_set(key, n_keys, uniq, part);
  for (int i = threadIdx.x; i < n; i += blockDim.x)
    if (uniq[i] < d.n_if) atomicAdd(&n_inner, 1);
  __syncthreads();
  if constexpr (!FILL) {
    if (threadIdx.x == 0) {
      counts[2 * blockIdx.x] = n_inner;
      counts[2 * blockIdx.x + 1] = n - n_inner;
    }
  } else {
    constexpr int kQ = kFace * static_cast<int>(sizeof(C)) / 16;
    const int f0 = first[blockIdx.x], b0 = bfirst[blockIdx.x];
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      if (i < n_inner) {
        face[f0 + i] = uniq[i];
        const V* src = reinterpret_cast<const V*>(d.face + static_cast<long long>(uniq[i]) * kFace);
        for (int q = 0; q < kQ; ++q)
          rec[static_cast<long long>(kQ) * f0 + static_cast<long long>(q) * n_inner + i] = src[q];
      } else {
        bface[b0 + i - n_inner] = uniq[i] - d.n_if;
      }
    }
    if (c < d.n) {
      const long long out = inc_start[c >> 5] + (c & 31);
      for (int j = 0; j < il; j += 4) {
        unsigned v[4] = {0u, 0u, 0u, 0u};
        for (int k = 0; k < 4 && j + k < il; ++k) {
          const int code = d.inc_code[base + static_cast<long long>(j + k) * kSlice];
          v[k] = 2u * static_cast<unsigned>(place_of(uniq, n, key_of(code))) +
                 (code >= 0 && (code & 1) ? 1u : 0u);
        }
        inc[out + static_cast<long long>(j / 4) * kSlice] = make_uint2(v[0] | (v[1] << 16), v[2] | (v[3] << 16));
      }
    }
  }
}

// The flux of every face of a block into shared memory (5 words a face), then each of its cells adds
// its own in increasing face index and takes its RK stage (finish_cell), then the next boundary
// states of its boundary faces: the work of k_face_flux, k_bface_flux, k_gather and the next stage's
// k_boundary_states in one launch, with the same operations in the same order. Faces between two
// blocks are computed in both; no flux goes through global memory. blockDim.x is the block's cells
// or, where the cells alone do not fill the chip, a multiple: its faces then take fewer rounds. Dynamic
// shared memory: 5 words per face of the largest block (and per cell). On small meshes it is bound by one
// round of dependent loads and the flux arithmetic of a face or two a thread: the 31 154-cell channel's
// stage takes 15 us where the four launches took 35. On large ones it computes a quarter of the interior
// faces twice (1.27 computations a face at 128 cells a block in Morton order), which costs more than the
// fluxes' way through memory (choose_defaults has the line); 230 880 cells: 43 us, stalled on the loads of
// the cells' records (39 % of the warps resident), against 41 for flux and gather. Registers bounded for
// four blocks of 256 per SM: 769 us a step's faces on the 1 942 000-cell channel, for three 858, for
// five 880.
template <class P, bool PLANAR, bool SECOND>
constexpr int kFaceBlockMin = sizeof(typename P::C) == 4 ? ((PLANAR || !SECOND) ? 4 : 3) : (SECOND ? 1 : 2);
template <class P, int FLUX, bool PLANAR, bool SECOND>
__global__ void __launch_bounds__(256, (kFaceBlockMin<P, PLANAR, SECOND>))
    k_faces_block(Dev<P> d, FaceBlocks<P> g, int mode, int stage, double wa, double wb, int local,
                  int last) {
  using C = typename P::C;
  using V = typename P::V;
  constexpr int kQ = kFace * static_cast<int>(sizeof(C)) / 16;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  C* const flux = reinterpret_cast<C*>(smem_raw);
  const int b = g.active != nullptr ? __ldg(g.active + blockIdx.x) : static_cast<int>(blockIdx.x);
  const int t = threadIdx.x, nt = blockDim.x, nb = g.cells;
  const int c = t < nb ? b * nb + t : d.n;  // threads past the cells only take faces
  const int f0 = __ldg(g.first + b), nf = __ldg(g.first + b + 1) - f0;
  const int b0 = __ldg(g.bfirst + b), nbf = __ldg(g.bfirst + b + 1) - b0;
  const V* const rec = g.rec + static_cast<long long>(kQ) * f0;
  int il = 0;
  double vol = 1.0;
  uint2 places = make_uint2(0u, 0u);
  const uint2* inc = g.inc;
  if (c < d.n) {
    il = __ldg(d.inc_len + c);
    vol = __ldg(d.volume + c);
    inc += __ldg(g.inc_start + (c >> 5)) + (c & 31);
    if (il > 0) places = __ldg(inc);
  }
  dependents_may_start();
  previous_done();
  for (int i = t; i < nf + nbf; i += nt) {
    C out[5];
    if (i < nf) {
      C fr[kFace], wl[5], gl[15], pl[5], wr[5], gr[15], pr[5];
#pragma unroll
      for (int q = 0; q < kQ; ++q) {
        const V v = __ldg(rec + static_cast<long long>(q) * nf + i);
        if constexpr (P::kVec == 4) {
          fr[4 * q] = v.x, fr[4 * q + 1] = v.y, fr[4 * q + 2] = v.z, fr[4 * q + 3] = v.w;
        } else {
          fr[2 * q] = v.x, fr[2 * q + 1] = v.y;
        }
      }
      if (!cell_active(d, index_of(fr[7]))) continue;
      cell_recon<P, SECOND, true>(d, index_of(fr[7]), wl, pl, gl);
      cell_recon<P, SECOND, true>(d, index_of(fr[11]), wr, pr, gr);
      const int f = PLANAR ? 0 : __ldg(g.face + f0 + i);
      interior_flux<P, FLUX, PLANAR>(d, f, fr, wl, gl, pl, wr, gr, pr, out);
    } else {
      const int bf = __ldg(g.bface + b0 + i - nf);
      C br[kBface], wc[5], gc[15], pc[5];
      load_words<P, true>(d.bface + static_cast<long long>(bf) * kBface, 0, kBface, br);
      if (!cell_active(d, index_of(br[13]))) continue;
      cell_recon<P, SECOND, true>(d, index_of(br[13]), wc, pc, gc);
      boundary_flux<P, FLUX, PLANAR>(d, bf, br, wc, gc, pc, out);
    }
#pragma unroll
    for (int k = 0; k < 5; ++k) flux[5 * i + k] = out[k];
  }
  const bool live = c < d.n && cell_active(d, c);
  CellIn in;
  if (live) load_cell_in(d, c, mode, stage, local, in);
  __syncthreads();
  C w[5] = {C(0), C(0), C(0), C(0), C(0)};
  if (live) {
    double res[5];
    const C nv = -static_cast<C>(vol);  // sources (:611-616): res = -V s
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      const C s = d.source != nullptr ? __ldg(d.source + static_cast<long long>(k) * d.n + c) : C(0.0);
      res[k] = mode == kFaceParts ? 0.0 : static_cast<double>(nv * s);  // face_parts: from zero
    }
    for (int j0 = 0; j0 < il; j0 += 4) {
      const uint2 next = j0 + 4 < il ? __ldg(inc + static_cast<long long>(j0 / 4 + 1) * kSlice) : places;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (j0 + q < il) {
          const unsigned v = q < 2 ? places.x : places.y;
          const unsigned place = q & 1 ? v >> 16 : v & 0xffffu;
          const C* fv = flux + 5 * (place >> 1);
          if (place & 1u) {
#pragma unroll
            for (int k = 0; k < 5; ++k) res[k] -= static_cast<double>(fv[k]);
          } else {
#pragma unroll
            for (int k = 0; k < 5; ++k) res[k] += static_cast<double>(fv[k]);
          }
        }
      }
      places = next;
    }
    finish_cell(d, c, res, vol, mode, stage, wa, wb, last, in, true, w);
  }
  if (g.wfirst != nullptr && (mode == kRk3 || mode == kRk4)) {
    const int w0 = __ldg(g.wfirst + b), nw = __ldg(g.wfirst + b + 1) - w0;
    if (nw == 0) return;
    __syncthreads();  // every cell has read its fluxes
#pragma unroll
    for (int k = 0; k < 5; ++k)
      if (t < nb) flux[5 * t + k] = w[k];
    __syncthreads();
    C* const next_b = d.prim_next + (d.prim_b - d.prim);
    for (int i = t; i < nw; i += nt) {
      const int bf = __ldg(g.walls + w0 + i);
      C r[kBface], wo[5], out[8];
      load_words<P, true>(d.bface + static_cast<long long>(bf) * kBface, 0, kBface, r);
      const int o = index_of(r[13]);
      if (!cell_active(d, o)) continue;
#pragma unroll
      for (int k = 0; k < 5; ++k) wo[k] = flux[5 * (o - b * nb) + k];
      boundary_value(wo, r[7], r + 8, r, d.p, out);
      out[5] = out[6] = out[7] = C(0);
      store_words<P, true>(next_b + static_cast<long long>(bf) * kPrimB, 0, 8, out);
      note_special(out, d.ctl);
    }
  }
}
