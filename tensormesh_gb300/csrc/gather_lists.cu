// Lists of the element-once assembly (gather.cuh), built from the connectivity
// and the slot map of the CSR pattern: the incidences of every node
//
//   nptr, nrec   e * B + a of every incidence of a node, ascending
//
// for P2 meshes, per node-level CSR position
//
//   ent[t]   kDiag, or the start of its list of records (a position below the
//            diagonal names its mirror's list)
//   rec[]    per position above the diagonal, contiguous: one record per
//            element that holds the node pair, elements ascending, the last
//            one marked
//
// and, for P1 meshes, the groups of rows described below.  Count, scan (by the
// caller), fill with integer atomics, then a sort of every short list, so the
// result does not depend on the order the atomics resolve in.
#include "gather.cuh"

namespace tmg {
namespace ga {

// local pair (a, b), a < b, of pair index k
TM_D void pair_nodes(int k, int B, int& a, int& b) {
  a = 0;
  int left = B - 1;
  while (k >= left) {
    k -= left;
    ++a;
    --left;
  }
  b = a + 1 + k;
}

__global__ void list_count_kernel(const int32_t* __restrict__ el, int64_t n, int B, int P,
                                  const int64_t* __restrict__ slots, int32_t* __restrict__ cnt, int32_t* bad) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;  // element * P + pair
  if (i >= n) return;
  const int64_t e = i / P;
  int a, b;
  pair_nodes((int)(i - e * P), B, a, b);
  const int va = el[e * B + a], vb = el[e * B + b];
  if (va == vb) {
    atomicExch(bad, 1);  // a repeated node: the caller keeps the patch kernels
    return;
  }
  const int64_t s = va < vb ? slots[(e * B + a) * B + b] : slots[(e * B + b) * B + a];
  atomicAdd(cnt + s, 1);
}

__global__ void list_fill_kernel(const int32_t* __restrict__ el, int64_t n, int B, int P,
                                 const int64_t* __restrict__ slots, const int64_t* __restrict__ start,
                                 int32_t* __restrict__ cnt, uint32_t* __restrict__ ent, uint32_t* __restrict__ rec) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t e = i / P;
  const int k = (int)(i - e * P);
  int a, b;
  pair_nodes(k, B, a, b);
  const bool flip = el[e * B + a] > el[e * B + b];
  const int64_t sab = slots[(e * B + a) * B + b], sba = slots[(e * B + b) * B + a];
  const int64_t up = flip ? sba : sab, low = flip ? sab : sba;
  const uint32_t s0 = (uint32_t)start[up];
  // every element of the pair writes the same entry words
  ent[up] = s0;
  ent[low] = s0 | kLower;
  if (b == a + 1) {
    ent[slots[(e * B + a) * B + a]] = kDiag;
    if (b == B - 1) ent[slots[(e * B + b) * B + b]] = kDiag;
  }
  const int at = atomicSub(cnt + up, 1) - 1;
  rec[s0 + at] = (uint32_t)i | (flip ? kFlip : 0u);
}

// Sorts every list and marks its last record.  A list's length is the gap to
// the next list's start.
__global__ void list_sort_kernel(int64_t nnz, const int64_t* __restrict__ start, uint32_t* __restrict__ rec) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= nnz) return;
  const int64_t s0 = start[t], s1 = start[t + 1];
  if (s1 == s0) return;
  for (int64_t i = s0 + 1; i < s1; ++i) {
    const uint32_t v = rec[i];
    int64_t j = i;
    while (j > s0 && (rec[j - 1] & kIdx) > (v & kIdx)) {
      rec[j] = rec[j - 1];
      --j;
    }
    rec[j] = v;
  }
  rec[s1 - 1] |= kEnd;
}

__global__ void node_count_kernel(const int32_t* __restrict__ el, int64_t n, int32_t* __restrict__ cnt) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) atomicAdd(cnt + el[i], 1);
}
__global__ void node_fill_kernel(const int32_t* __restrict__ el, int64_t n, const int64_t* __restrict__ nptr,
                                 int32_t* __restrict__ cnt, uint32_t* __restrict__ nrec) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int v = el[i];
  nrec[nptr[v] + atomicSub(cnt + v, 1) - 1] = (uint32_t)i;
}
__global__ void node_sort_kernel(int64_t n_points, const int64_t* __restrict__ nptr, uint32_t* __restrict__ nrec) {
  const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (r >= n_points) return;
  const int64_t s0 = nptr[r], s1 = nptr[r + 1];
  for (int64_t i = s0 + 1; i < s1; ++i) {
    const uint32_t v = nrec[i];
    int64_t j = i;
    while (j > s0 && nrec[j - 1] > v) {
      nrec[j] = nrec[j - 1];
      --j;
    }
    nrec[j] = v;
  }
}

// ---- groups of P1 rows -------------------------------------------------------
// A group is `rows_per_group` consecutive entries of a node order that follows
// the space (a Z-order curve), so that its rows share elements.  Per group:
// its distinct elements (ascending), and per CSR entry of its rows a word
// (record start | local row << 16, kDiag on the diagonal) and the list of
// 16-bit records, elements ascending:
//   scalar  local element * pairs + pair, in quads: the start counts quads, pad
//           records name a zero (local element = number of elements, pair 0)
//           and bit 15 of a quad's fourth record marks the last quad
//   block   local element << 4 | a << 2 | b (row node = local node a, column
//           node = b), bit 15 on the last record
constexpr int kGroupThreads = 256;
constexpr int kGroupInc = 4096;    // incidences of one group's rows

// Sorted distinct elements of group g in s_e[0, n); returns n, or -1 when the
// group holds too many incidences.  s_off[k]: incidences before row k.
TM_D int group_elements(int g, int rows_per_group, int n_points, int B, const int32_t* __restrict__ order,
                        const int64_t* __restrict__ nptr, const uint32_t* __restrict__ nrec, int* s_e, int* s_off,
                        int* s_scan) {
  const int tid = threadIdx.x;
  const int r0 = g * rows_per_group, nr = min(rows_per_group, n_points - r0);
  if (tid < nr) {
    const int r = order[r0 + tid];
    s_off[tid + 1] = (int)(nptr[r + 1] - nptr[r]);
  }
  __syncthreads();
  if (tid == 0) {
    s_off[0] = 0;
    for (int k = 0; k < nr; ++k) s_off[k + 1] = min(s_off[k] + s_off[k + 1], kGroupInc + 1);
  }
  __syncthreads();
  const int total = s_off[nr];
  if (total > kGroupInc) return -1;
  int n2 = 32;
  while (n2 < total) n2 <<= 1;
  for (int k = tid >> 5; k < nr; k += kGroupThreads / 32) {
    const int64_t b = nptr[order[r0 + k]];
    for (int i = s_off[k] + (tid & 31); i < s_off[k + 1]; i += 32) s_e[i] = (int)(nrec[b + i - s_off[k]] / (uint32_t)B);
  }
  for (int i = total + tid; i < n2; i += kGroupThreads) s_e[i] = 0x7fffffff;
  __syncthreads();
  for (int size = 2; size <= n2; size <<= 1)
    for (int st = size >> 1; st > 0; st >>= 1) {
      for (int i = tid; i < n2 / 2; i += kGroupThreads) {
        const int lo = 2 * i - (i & (st - 1)), hi = lo + st;
        const bool up = (lo & size) == 0;
        const int x = s_e[lo], y = s_e[hi];
        if ((x > y) == up) {
          s_e[lo] = y;
          s_e[hi] = x;
        }
      }
      __syncthreads();
    }
  // distinct values, each thread a contiguous run of at most 16
  const int per = (n2 + kGroupThreads - 1) / kGroupThreads, i0 = tid * per;
  int vals[kGroupInc / kGroupThreads], c = 0;
  for (int i = i0; i < min(i0 + per, total); ++i)
    if (i == 0 || s_e[i] != s_e[i - 1]) vals[c++] = s_e[i];
  s_scan[tid] = c;
  __syncthreads();
  for (int o = 1; o < kGroupThreads; o <<= 1) {
    const int v = tid >= o ? s_scan[tid - o] : 0;
    __syncthreads();
    s_scan[tid] += v;
    __syncthreads();
  }
  const int n = s_scan[kGroupThreads - 1];
  for (int i = 0; i < c; ++i) s_e[s_scan[tid] - c + i] = vals[i];
  __syncthreads();
  return n;
}

// Records that a list of c elements takes
TM_D int list_slots(int c, bool quads) { return quads ? (c + 3) & ~3 : c; }

// Sizes of every group: [distinct elements, CSR entries, records]; *bad is
// raised where the 16-bit forms do not hold them.
__global__ void __launch_bounds__(kGroupThreads)
group_count_kernel(int rows_per_group, int n_points, int B, int quads, const int32_t* __restrict__ order,
                   const int64_t* __restrict__ nptr, const uint32_t* __restrict__ nrec,
                   const int64_t* __restrict__ indptr, const int64_t* __restrict__ slots,
                   int32_t* __restrict__ cnt, int32_t* __restrict__ sizes, int32_t* bad) {
  __shared__ int s_e[kGroupInc];
  __shared__ int s_off[kGroupRows + 1];
  __shared__ int s_scan[kGroupThreads];
  __shared__ int s_sum[2];
  const int g = blockIdx.x, tid = threadIdx.x;
  if (tid < 2) s_sum[tid] = 0;
  const int n = group_elements(g, rows_per_group, n_points, B, order, nptr, nrec, s_e, s_off, s_scan);
  const int r0 = g * rows_per_group, nr = min(rows_per_group, n_points - r0);
  if (n >= 0 && tid < nr) {
    const int r = order[r0 + tid];
    const int64_t c0 = indptr[r];
    const int deg = (int)(indptr[r + 1] - c0);
    int32_t* c = cnt + c0;   // list lengths of the row (used again by the fill pass)
    for (int p = 0; p < deg; ++p) c[p] = 0;
    for (int64_t i = nptr[r]; i < nptr[r + 1]; ++i) {
      const int64_t row = (int64_t)nrec[i] * B;   // slots of (element, a)
      const int a = (int)(nrec[i] % (uint32_t)B);
      for (int b = 0; b < B; ++b)
        if (b != a) ++c[slots[row + b] - c0];
    }
    int recs = 0;
    for (int p = 0; p < deg; ++p) recs += list_slots(c[p], quads);
    atomicAdd(s_sum, deg);
    atomicAdd(s_sum + 1, recs);
  }
  __syncthreads();
  if (tid != 0) return;
  const bool over = n < 0 || s_sum[0] > (quads ? 65535 : kBlockEntries) ||
                    (quads ? (n * (B * (B - 1) / 2) > kPairValues || s_sum[1] / 4 > 65535)
                           : (n > kBlockElems || s_sum[1] > 65535));
  if (over) atomicExch(bad, 1);
  sizes[3 * g] = over ? 0 : n;
  sizes[3 * g + 1] = over ? 0 : s_sum[0];
  sizes[3 * g + 2] = over ? 0 : s_sum[1];
}

__global__ void __launch_bounds__(kGroupThreads)
group_fill_kernel(int rows_per_group, int n_points, int B, int quads, const int32_t* __restrict__ order,
                  const int64_t* __restrict__ nptr, const uint32_t* __restrict__ nrec,
                  const int64_t* __restrict__ indptr, const int64_t* __restrict__ slots, int32_t* __restrict__ cnt,
                  const int64_t* __restrict__ base, int32_t* __restrict__ gelem, uint32_t* __restrict__ gent,
                  uint16_t* __restrict__ grec) {
  __shared__ int s_e[kGroupInc];
  __shared__ int s_off[kGroupRows + 1];
  __shared__ int s_scan[kGroupThreads];
  __shared__ int s_ent[kGroupRows + 1], s_rec[kGroupRows + 1];
  const int g = blockIdx.x, tid = threadIdx.x;
  const int n = group_elements(g, rows_per_group, n_points, B, order, nptr, nrec, s_e, s_off, s_scan);
  const int r0 = g * rows_per_group, nr = min(rows_per_group, n_points - r0);
  for (int i = tid; i < n; i += kGroupThreads) gelem[base[3 * g] + i] = s_e[i];
  const bool on = tid < nr;
  int r = 0, deg = 0;
  int64_t c0 = 0;
  if (on) {
    r = order[r0 + tid];
    c0 = indptr[r];
    deg = (int)(indptr[r + 1] - c0);
    int recs = 0;
    for (int p = 0; p < deg; ++p) recs += list_slots(cnt[c0 + p], quads);
    s_ent[tid + 1] = deg;
    s_rec[tid + 1] = recs;
  }
  __syncthreads();
  if (tid == 0) {
    s_ent[0] = s_rec[0] = 0;
    for (int k = 0; k < nr; ++k) {
      s_ent[k + 1] += s_ent[k];
      s_rec[k + 1] += s_rec[k];
    }
  }
  __syncthreads();
  if (!on) return;
  uint16_t* rec = grec + base[3 * g + 2];
  uint32_t* ent = gent + base[3 * g + 1] + s_ent[tid];
  const int P = B * (B - 1) / 2;
  int at = s_rec[tid];
  for (int p = 0; p < deg; ++p) {
    const int c = cnt[c0 + p], w = list_slots(c, quads);
    ent[p] = c ? (uint32_t)(quads ? at / 4 : at) | ((uint32_t)tid << 16) : kDiag;
    for (int k = c; k < w; ++k) rec[at + k] = (uint16_t)(n * P | (k == w - 1 ? 0x8000 : 0));   // zeros
    cnt[c0 + p] = at;
    at += w;
  }
  // records in element order; the cursor of a list stops at its last record
  for (int64_t i = nptr[r]; i < nptr[r + 1]; ++i) {
    const uint32_t e = nrec[i] / (uint32_t)B;
    const int64_t row = (int64_t)nrec[i] * B;
    const int a = (int)(nrec[i] - e * B);
    int lo = 0, hi = n;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (s_e[mid] < (int)e) lo = mid + 1; else hi = mid;
    }
    for (int b = 0; b < B; ++b) {
      if (b == a) continue;
      const int p = (int)(slots[row + b] - c0);
      const int x = a < b ? a : b, y = a < b ? b : a;
      const int code = quads ? lo * P + x * (2 * B - x - 1) / 2 + (y - x - 1) : (lo << 4) | (a << 2) | b;
      const int k = cnt[c0 + p]++;
      // the end of this list's slots: the start of the next list, or of the next row's
      int next = s_rec[tid + 1];
      for (int q = p + 1; q < deg; ++q)
        if (ent[q] != kDiag) {
          next = (int)(ent[q] & 0xffffu) * (quads ? 4 : 1);
          break;
        }
      rec[k] = (uint16_t)(code | (k == next - 1 ? 0x8000 : 0));
    }
  }
}

}  // namespace ga
}  // namespace tmg

extern "C" int tm_gather_count(const int32_t* elements, int64_t n_elements, int32_t n_basis, int64_t nnz,
                               const int64_t* slots, int32_t* cnt, int32_t* bad, void* stream) {
  if (n_elements < 0 || n_basis < 2 || nnz < 0 || !cnt || !bad) return TM_ERR_INVALID;
  if (n_elements > 0 && (!elements || !slots)) return TM_ERR_INVALID;
  const int P = n_basis * (n_basis - 1) / 2;
  if (n_elements * P >= (int64_t)tmg::ga::kIdx) return TM_ERR_INDEX;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (cudaMemsetAsync(cnt, 0, sizeof(int32_t) * nnz, s) != cudaSuccess) return TM_ERR_CUDA;
  if (cudaMemsetAsync(bad, 0, sizeof(int32_t), s) != cudaSuccess) return TM_ERR_CUDA;
  const int64_t n = n_elements * P;
  if (n > 0)
    tmg::ga::list_count_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(elements, n, n_basis, P, slots, cnt, bad);
  return cudaPeekAtLastError() == cudaSuccess ? TM_OK : TM_ERR_CUDA;
}

extern "C" int tm_gather_fill(const int32_t* elements, int64_t n_elements, int32_t n_basis, int64_t nnz,
                              const int64_t* slots, const int64_t* start, int32_t* cnt, uint32_t* ent, uint32_t* rec,
                              void* stream) {
  if (n_elements < 0 || n_basis < 2 || nnz < 0) return TM_ERR_INVALID;
  if (n_elements == 0 || nnz == 0) return TM_OK;
  if (!elements || !slots || !start || !cnt || !ent || !rec) return TM_ERR_INVALID;
  const int P = n_basis * (n_basis - 1) / 2;
  if (n_elements * P >= (int64_t)tmg::ga::kIdx) return TM_ERR_INDEX;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int64_t n = n_elements * P;
  tmg::ga::list_fill_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(elements, n, n_basis, P, slots, start, cnt,
                                                                        ent, rec);
  tmg::ga::list_sort_kernel<<<(unsigned)((nnz + 255) / 256), 256, 0, s>>>(nnz, start, rec);
  return cudaPeekAtLastError() == cudaSuccess ? TM_OK : TM_ERR_CUDA;
}

extern "C" int tm_node_lists(const int32_t* elements, int64_t n_elements, int32_t n_basis, int64_t n_points,
                             const int64_t* nptr, int32_t* cnt, uint32_t* nrec, void* stream) {
  if (n_elements < 0 || n_basis < 1 || n_points < 0 || !cnt) return TM_ERR_INVALID;
  if (n_elements * n_basis >= (int64_t)0x7fffffff) return TM_ERR_INDEX;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int64_t n = n_elements * n_basis;
  if (n > 0 && !elements) return TM_ERR_INVALID;
  const unsigned grid = (unsigned)((n + 255) / 256);
  if (!nptr) {  // first call: incidences per node
    if (cudaMemsetAsync(cnt, 0, sizeof(int32_t) * n_points, s) != cudaSuccess) return TM_ERR_CUDA;
    if (n > 0) tmg::ga::node_count_kernel<<<grid, 256, 0, s>>>(elements, n, cnt);
  } else if (n > 0) {
    if (!nrec) return TM_ERR_INVALID;
    tmg::ga::node_fill_kernel<<<grid, 256, 0, s>>>(elements, n, nptr, cnt, nrec);
    tmg::ga::node_sort_kernel<<<(unsigned)((n_points + 255) / 256), 256, 0, s>>>(n_points, nptr, nrec);
  }
  return cudaPeekAtLastError() == cudaSuccess ? TM_OK : TM_ERR_CUDA;
}

extern "C" int tm_group_count(int32_t n_basis, int64_t n_points, int32_t rows_per_group, int32_t quads,
                              const int32_t* order, const int64_t* nptr, const uint32_t* nrec, const int64_t* indptr,
                              const int64_t* slots, int32_t* cnt, int32_t* sizes, int32_t* bad, void* stream) {
  if (n_basis < 2 || n_basis > 4 || n_points < 0 || rows_per_group < 1 || rows_per_group > tmg::ga::kGroupRows)
    return TM_ERR_INVALID;
  if (!order || !nptr || !nrec || !indptr || !slots || !cnt || !sizes || !bad) return TM_ERR_INVALID;
  if (n_points >= (int64_t)0x7fffffff) return TM_ERR_INDEX;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (cudaMemsetAsync(bad, 0, sizeof(int32_t), s) != cudaSuccess) return TM_ERR_CUDA;
  const int64_t g = (n_points + rows_per_group - 1) / rows_per_group;
  if (g > 0)
    tmg::ga::group_count_kernel<<<(unsigned)g, tmg::ga::kGroupThreads, 0, s>>>(
        rows_per_group, (int)n_points, n_basis, quads, order, nptr, nrec, indptr, slots, cnt, sizes, bad);
  return cudaPeekAtLastError() == cudaSuccess ? TM_OK : TM_ERR_CUDA;
}

extern "C" int tm_group_fill(int32_t n_basis, int64_t n_points, int32_t rows_per_group, int32_t quads,
                             const int32_t* order, const int64_t* nptr, const uint32_t* nrec, const int64_t* indptr,
                             const int64_t* slots, int32_t* cnt, const int64_t* base, int32_t* gelem, uint32_t* gent,
                             uint16_t* grec, void* stream) {
  if (n_basis < 2 || n_basis > 4 || n_points < 0 || rows_per_group < 1 || rows_per_group > tmg::ga::kGroupRows)
    return TM_ERR_INVALID;
  if (!order || !nptr || !nrec || !indptr || !slots || !cnt || !base || !gelem || !gent || !grec) return TM_ERR_INVALID;
  if (n_points >= (int64_t)0x7fffffff) return TM_ERR_INDEX;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int64_t g = (n_points + rows_per_group - 1) / rows_per_group;
  if (g > 0)
    tmg::ga::group_fill_kernel<<<(unsigned)g, tmg::ga::kGroupThreads, 0, s>>>(
        rows_per_group, (int)n_points, n_basis, quads, order, nptr, nrec, indptr, slots, cnt, base, gelem, gent, grec);
  return cudaPeekAtLastError() == cudaSuccess ? TM_OK : TM_ERR_CUDA;
}
