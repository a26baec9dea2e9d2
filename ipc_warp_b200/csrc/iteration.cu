// The two ends of a contact iteration as one launch each: everything that has
// to be reset or formed before the queries, and the results written straight
// into the host's pinned words.  Ten fills and copies of a few bytes took
// about 2 us each at the two ends of a 160 us iteration of a small scene.
#include "common.cuh"

namespace ipcb {
int check_launch(const char* where);

namespace {

template <class S>
__global__ void k_begin(const S* __restrict__ x, const S* __restrict__ dx, S* __restrict__ x1, S* __restrict__ b,
                        int n3, int* ee_cnt, int* pt_cnt, int* status, int* bsr_status, double* energy, S* toi,
                        float4* __restrict__ x4) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n3) {
    b[i] = S(0);
    if (dx) x1[i] = xsub(x[i], dx[i]);
  }
  if (3 * i < n3) x4[i] = make_float4((float)x[3 * i], (float)x[3 * i + 1], (float)x[3 * i + 2], 0.f);
  if (i == 0) {
    *ee_cnt = *pt_cnt = *status = *bsr_status = 0;
    *energy = 0.0;
    *toi = S(1);
  }
}

template <class S>
__global__ void k_results(const int* ee_cnt, const int* pt_cnt, const int* bsr_status, const int* status,
                          const double* energy, const S* toi, int* counts_out, double* energy_out, S* toi_out) {
  counts_out[0] = *ee_cnt;
  counts_out[1] = *pt_cnt;
  counts_out[2] = *bsr_status;
  counts_out[3] = *status;
  *energy_out = *energy;
  *toi_out = *toi;
}

constexpr int kMaxWords = 8;
struct Words {
  int* dst[kMaxWords];
  const int* src[kMaxWords];
};

__global__ void k_words(Words w, int n) {
  const int i = threadIdx.x;
  if (i < n) *w.dst[i] = w.src[i] ? *w.src[i] : 0;
}

}  // namespace
}  // namespace ipcb

using namespace ipcb;

extern "C" {

int ipcb_iteration_begin(const ipcb_soup* soup, const void* dx, void* x1, void* b, int* ee_cnt, int* pt_cnt,
                         int* status, int* bsr_status, double* energy, void* toi, float* x4, ipcb_stream s) {
  if (!soup || !b || (dx && !x1) || !ee_cnt || !pt_cnt || !status || !bsr_status || !energy || !toi || !x4)
    return IPCB_E_ARG;
  const int n3 = 3 * soup->n_verts, grid = div_up(n3 > 0 ? n3 : 1, 256);
  if (soup->fp64)
    k_begin<double><<<grid, 256, 0, (cudaStream_t)s>>>((const double*)soup->x, (const double*)dx, (double*)x1,
                                                       (double*)b, n3, ee_cnt, pt_cnt, status, bsr_status, energy,
                                                       (double*)toi, (float4*)x4);
  else
    k_begin<float><<<grid, 256, 0, (cudaStream_t)s>>>((const float*)soup->x, (const float*)dx, (float*)x1, (float*)b,
                                                      n3, ee_cnt, pt_cnt, status, bsr_status, energy, (float*)toi,
                                                      (float4*)x4);
  return check_launch("ipcb_iteration_begin");
}

int ipcb_iteration_results(int fp64, const int* ee_cnt, const int* pt_cnt, const int* bsr_status, const int* status,
                           const double* energy, const void* toi, int* counts_out, double* energy_out, void* toi_out,
                           ipcb_stream s) {
  if (!ee_cnt || !pt_cnt || !bsr_status || !status || !energy || !toi || !counts_out || !energy_out || !toi_out)
    return IPCB_E_ARG;
  if (fp64)
    k_results<double><<<1, 1, 0, (cudaStream_t)s>>>(ee_cnt, pt_cnt, bsr_status, status, energy, (const double*)toi,
                                                    counts_out, energy_out, (double*)toi_out);
  else
    k_results<float><<<1, 1, 0, (cudaStream_t)s>>>(ee_cnt, pt_cnt, bsr_status, status, energy, (const float*)toi,
                                                   counts_out, energy_out, (float*)toi_out);
  return check_launch("ipcb_iteration_results");
}

// Counters are a few words in as many arrays: a fill or a copy of each is a
// launch of 1.5 to 3 us and 5 to 10 us of host time.
int ipcb_words(int n, void* const* dst, const void* const* src, ipcb_stream s) {
  if (n < 0 || n > kMaxWords || !dst || !src) return IPCB_E_ARG;
  if (n == 0) return IPCB_OK;
  Words w{};
  for (int i = 0; i < n; ++i) {
    if (!dst[i]) return IPCB_E_ARG;
    w.dst[i] = (int*)dst[i];
    w.src[i] = (const int*)src[i];
  }
  k_words<<<1, 32, 0, (cudaStream_t)s>>>(w, n);
  return check_launch("ipcb_words");
}

}  // extern "C"
