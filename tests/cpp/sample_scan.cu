// The grid sampling of one coupling (sample_grid) on given PDFs, for tests/test_gpu_sampling.py: the
// coupling matrix is diag(1, -1, 0, 0), so that a grid point (a, b, 0, 0) has C x x = a^2 - b^2.
#define MQ_DEVICE_ONLY
#include "walker_general.cuh"

namespace {

__global__ void scan_kernel(mq::Dev p, const double *grids, double ov, int *index, double *factor) {
  __shared__ double M[16], Cm[16], O1[4], O2[4], sc[16], id[16], one[4], pdf[1024];
  mq::Smem s{};
  s.M = M;
  s.Cm = Cm;
  s.O1 = O1;
  s.O2 = O2;
  s.sc = sc;
  s.pdf = pdf;
  s.tabU = s.tabVT = id;
  s.tabSq = one;
  s.grid = grids + 4L * p.G * blockIdx.x;
  s.w = blockIdx.x;
  if (threadIdx.x < 16) {
    id[threadIdx.x] = threadIdx.x % 5 == 0 ? 1.0 : 0.0;
    M[threadIdx.x] = threadIdx.x == 0 ? 1.0 : threadIdx.x == 5 ? -1.0 : 0.0;
    if (threadIdx.x < 4) one[threadIdx.x] = 1.0;
    sc[threadIdx.x] = 1.0;
  }
  if (threadIdx.x == 0) sc[mq::kScOv] = ov;
  __syncthreads();
  mq::sample_grid<double>(p, s, 0, 0);
  if (threadIdx.x == 0) {
    index[blockIdx.x] = (int)sc[2];
    factor[blockIdx.x] = sc[4];
  }
}

}  // namespace

// n samplings: grids [n][G][4], one uniform each; the index and the weight factor (sum of the PDF) out.
extern "C" int sample_scan(int n, int G, int threads, double ov, const double *grids, const double *u, int *index,
                           double *factor) {
  double *g = nullptr, *ud = nullptr, *f = nullptr;
  int *ix = nullptr;
  if (G > 992 || cudaMalloc(&g, sizeof(double) * 4 * n * G) || cudaMalloc(&ud, sizeof(double) * n) ||
      cudaMalloc(&f, sizeof(double) * n) || cudaMalloc(&ix, sizeof(int) * n) ||
      cudaMemcpy(g, grids, sizeof(double) * 4 * n * G, cudaMemcpyHostToDevice) ||
      cudaMemcpy(ud, u, sizeof(double) * n, cudaMemcpyHostToDevice))
    return 1;
  mq::Dev p{};
  p.G = G;
  p.nC = 1;
  p.uni = ud;
  scan_kernel<<<n, threads>>>(p, g, ov, ix, f);
  const int rc = cudaMemcpy(index, ix, sizeof(int) * n, cudaMemcpyDeviceToHost) ||
                 cudaMemcpy(factor, f, sizeof(double) * n, cudaMemcpyDeviceToHost);
  cudaFree(g);
  cudaFree(ud);
  cudaFree(f);
  cudaFree(ix);
  return rc;
}
