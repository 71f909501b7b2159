// Aligned rows from gap-DP paths: AlignTwoMSAsGivenPath (MU/aligngivenpath.cpp:256)
// for the single-sequence profiles of the pairwise path.  Each edge of a
// path is one column: 'M' takes the next character of both sequences, 'D'
// the next of A against a gap in B, 'I' a gap in A against the next of B;
// the gap character is '-' (MUSCLE's MSA gap).  The characters are copied
// as given (ASCII bases or 0..3 codes alike).
//
// A warp takes 128 edges per step, each lane's source positions from a ballot
// prefix of the edges before it.  One warp per problem, or, where there are
// too few problems to fill the device that way, a CTA of 32, whose warps count
// their shares of the path first.
#include "mvg_internal.h"

namespace mvg {

// Edges [t0, t1) of one path on one warp, whose first takes character i of A
// and j of B; both move on.  Returns whether an edge was none, or past a
// sequence's end.  kSteps: steps of 32 edges whose loads are in flight.
template <int kSteps>
__device__ __forceinline__ bool rows_of(const uint8_t* __restrict__ A, int64_t la, const uint8_t* __restrict__ B,
                                        int64_t lb, const char* __restrict__ P, int64_t t0, int64_t t1,
                                        uint8_t* __restrict__ RA, uint8_t* __restrict__ RB, int64_t& i, int64_t& j) {
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  bool bad = false;
  for (; t0 < t1; t0 += 32 * kSteps) {
    char e[kSteps];
#pragma unroll
    for (int s = 0; s < kSteps; ++s) {
      const int64_t t = t0 + 32 * s + lane;
      e[s] = t < t1 ? P[t] : 'X';
    }
#pragma unroll
    for (int s = 0; s < kSteps; ++s) {
      const int64_t t = t0 + 32 * s + lane;
      const bool ia = e[s] == 'M' || e[s] == 'D', ib = e[s] == 'M' || e[s] == 'I';
      const unsigned ma = __ballot_sync(0xffffffffu, ia), mb = __ballot_sync(0xffffffffu, ib);
      const int64_t pa = i + __popc(ma & below), pb = j + __popc(mb & below);
      if (t < t1) {
        bad |= !ia && !ib;
        bad |= (ia && pa >= la) || (ib && pb >= lb);
        RA[t] = ia && pa < la ? A[pa] : (uint8_t)'-';
        RB[t] = ib && pb < lb ? B[pb] : (uint8_t)'-';
      }
      i += __popc(ma);
      j += __popc(mb);
    }
  }
  return bad;
}

// WARPS warps per problem: 1 (eight problems per CTA) or 32 (a CTA each).
template <int WARPS>
__global__ void __launch_bounds__(WARPS == 1 ? 256 : 1024)
    k_path_rows(const uint8_t* __restrict__ sa, const uint64_t* __restrict__ oa, const uint8_t* __restrict__ sb,
                const uint64_t* __restrict__ ob, int64_t nprob, const char* __restrict__ paths,
                const uint64_t* __restrict__ path_off, const int64_t* __restrict__ path_len,
                uint8_t* __restrict__ rows_a, uint8_t* __restrict__ rows_b, uint32_t* err) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t first = WARPS == 1 ? (int64_t)blockIdx.x * 8 + wid : blockIdx.x;
  const int64_t step = WARPS == 1 ? (int64_t)gridDim.x * 8 : gridDim.x;
  for (int64_t p = first; p < nprob; p += step) {
    const uint8_t* A = sa + oa[p];
    const uint8_t* B = sb + ob[p];
    const int64_t la = (int64_t)(oa[p + 1] - oa[p]), lb = (int64_t)(ob[p + 1] - ob[p]);
    const int64_t n = path_len[p];
    const char* P = paths + path_off[p];
    int64_t i = 0, j = 0, t0 = 0, t1 = n;  // characters of A and B consumed before t0
    if constexpr (WARPS > 1) {
      __shared__ int64_t s_a[WARPS], s_b[WARPS];
      const int64_t share = ((n + WARPS - 1) / WARPS + 31) & ~(int64_t)31;
      t0 = min(n, wid * share);
      t1 = min(n, t0 + share);
      int64_t ca = 0, cb = 0;
#pragma unroll 4
      for (int64_t t = t0 + lane; t < t1; t += 32) {
        const char e = P[t];
        ca += e == 'M' || e == 'D';
        cb += e == 'M' || e == 'I';
      }
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) {
        ca += __shfl_xor_sync(0xffffffffu, ca, d);
        cb += __shfl_xor_sync(0xffffffffu, cb, d);
      }
      __syncthreads();  // the last problem's counts are read
      if (lane == 0) {
        s_a[wid] = ca;
        s_b[wid] = cb;
      }
      __syncthreads();
      for (int w = 0; w < wid; ++w) {
        i += s_a[w];
        j += s_b[w];
      }
    }
    bool bad = false;
    if (WARPS == 1) {  // a rest of up to 32 edges, or a short path, in one step (100,000 of 30: 44 and 37 us)
      const int64_t rest = n > 32 ? min(n, (n + 95) / 128 * 128) : 0;
      bad = rows_of<4>(A, la, B, lb, P, 0, rest, rows_a + path_off[p], rows_b + path_off[p], i, j);
      bad |= rows_of<1>(A, la, B, lb, P, rest, n, rows_a + path_off[p], rows_b + path_off[p], i, j);
    } else {
      bad = rows_of<4>(A, la, B, lb, P, t0, t1, rows_a + path_off[p], rows_b + path_off[p], i, j);
    }
    if (wid % WARPS == WARPS - 1) bad |= i != la || j != lb;  // the path must consume both sequences
    if (__any_sync(0xffffffffu, bad) && lane == 0) set_error(err, kDevRange);
  }
}

}  // namespace mvg

using namespace mvg;

static Ctx* rows_ctx(mvg_handle h) { return reinterpret_cast<Ctx*>(h); }

extern "C" int mvg_path_rows_dev(mvg_handle h, const uint8_t* d_seq_a, const uint64_t* d_off_a, const uint8_t* d_seq_b,
                                 const uint64_t* d_off_b, int64_t nprob, const char* d_paths,
                                 const uint64_t* d_path_off, const int64_t* d_path_len, uint8_t* d_rows_a,
                                 uint8_t* d_rows_b) {
  if (!h || nprob < 0 ||
      (nprob && (!d_seq_a || !d_off_a || !d_seq_b || !d_off_b || !d_paths || !d_path_off || !d_path_len ||
                 !d_rows_a || !d_rows_b)))
    return report_error(MVG_ERR_ARG, "null argument");
  if (nprob == 0) return 0;
  Ctx* c = rows_ctx(h);
  MVG_CUDA_TRY(cudaSetDevice(c->device));
  MVG_CUDA_TRY(cudaMemsetAsync(c->d_err, 0, 4, c->stream));
  // Below four problems per SM a warp per problem leaves most of the device
  // idle: the call took 162 us for one path of 10,000 edges with a warp, 26
  // with a CTA, and for 600 of 4,000 edges 65 and 38.  From there on CTAs of
  // short paths cost more than they give (2,000 of 4,000 edges: 67 and 68 us,
  // of 300: 26 and 42).
  constexpr int64_t kCtaProblems = 608;
  if (nprob <= kCtaProblems)
    k_path_rows<32><<<(unsigned)nprob, 1024, 0, c->stream>>>(d_seq_a, d_off_a, d_seq_b, d_off_b, nprob, d_paths,
                                                             d_path_off, d_path_len, d_rows_a, d_rows_b, c->d_err);
  else
    k_path_rows<1><<<grid_for((uint64_t)nprob * 32, 256), 256, 0, c->stream>>>(
        d_seq_a, d_off_a, d_seq_b, d_off_b, nprob, d_paths, d_path_off, d_path_len, d_rows_a, d_rows_b, c->d_err);
  c->launches++;
  MVG_CUDA_TRY(cudaGetLastError());
  const int rc = check_device_error(c);
  if (rc == MVG_ERR_RANGE) return report_error(MVG_ERR_ARG, "a path does not consume exactly its two sequences");
  return rc;
}

extern "C" int mvg_path_rows(mvg_handle h, const uint8_t* seq_a, const uint64_t* off_a, const uint8_t* seq_b,
                             const uint64_t* off_b, int64_t nprob, const char* paths, const uint64_t* path_off,
                             const int64_t* path_len, uint8_t* rows_a, uint8_t* rows_b) {
  if (!h || nprob < 0 ||
      (nprob && (!seq_a || !off_a || !seq_b || !off_b || !paths || !path_off || !path_len || !rows_a || !rows_b)))
    return report_error(MVG_ERR_ARG, "null argument");
  if (nprob == 0) return 0;
  Ctx* c = rows_ctx(h);
  MVG_CUDA_TRY(cudaSetDevice(c->device));
  const uint64_t na = off_a[nprob], nb = off_b[nprob], np = path_off[nprob];
  Workspace& ws = c->ws;
  uint8_t* dsa = (uint8_t*)ws.get(c, 46, na + 16);
  uint8_t* dsb = (uint8_t*)ws.get(c, 47, nb + 16);
  uint64_t* doa = (uint64_t*)ws.get(c, 5, (nprob + 1) * 8);
  uint64_t* dob = (uint64_t*)ws.get(c, 6, (nprob + 1) * 8);
  char* dpa = (char*)ws.get(c, 9, np + 16);
  uint64_t* dpo = (uint64_t*)ws.get(c, 8, (nprob + 1) * 8);
  int64_t* dpl = (int64_t*)ws.get(c, 22, nprob * 8);
  uint8_t* dra = (uint8_t*)ws.get(c, 68, np + 16);
  uint8_t* drb = (uint8_t*)ws.get(c, 69, np + 16);
  if (!dsa || !dsb || !doa || !dob || !dpa || !dpo || !dpl || !dra || !drb)
    return report_error(MVG_ERR_NOMEM, "workspace allocation failed");
  MVG_CUDA_TRY(cudaMemcpyAsync(dsa, seq_a, na, cudaMemcpyHostToDevice, c->stream));
  MVG_CUDA_TRY(cudaMemcpyAsync(dsb, seq_b, nb, cudaMemcpyHostToDevice, c->stream));
  MVG_CUDA_TRY(cudaMemcpyAsync(doa, off_a, (nprob + 1) * 8, cudaMemcpyHostToDevice, c->stream));
  MVG_CUDA_TRY(cudaMemcpyAsync(dob, off_b, (nprob + 1) * 8, cudaMemcpyHostToDevice, c->stream));
  MVG_CUDA_TRY(cudaMemcpyAsync(dpa, paths, np, cudaMemcpyHostToDevice, c->stream));
  MVG_CUDA_TRY(cudaMemcpyAsync(dpo, path_off, (nprob + 1) * 8, cudaMemcpyHostToDevice, c->stream));
  MVG_CUDA_TRY(cudaMemcpyAsync(dpl, path_len, nprob * 8, cudaMemcpyHostToDevice, c->stream));
  int rc = mvg_path_rows_dev(h, dsa, doa, dsb, dob, nprob, dpa, dpo, dpl, dra, drb);
  if (rc) return rc;
  MVG_CUDA_TRY(cudaMemcpyAsync(rows_a, dra, np, cudaMemcpyDeviceToHost, c->stream));
  MVG_CUDA_TRY(cudaMemcpyAsync(rows_b, drb, np, cudaMemcpyDeviceToHost, c->stream));
  MVG_CUDA_TRY(cudaStreamSynchronize(c->stream));
  return 0;
}
