// sfm_refresh.cu — the landmark reprojection-error refresh that openmvg-sfm runs after it commits a
// bundle adjustment (refresh_landmark_reprojection_errors_for, crates/openmvg-sfm/src/ops/
// reconstruction/bundle.rs:510-637), on the GPU.
//
// One thread per landmark walks the landmark's track in order: for each supporting observation whose
// view has a pose it evaluates the pixel-equivalent residual of the camera residual policy with no
// limit (camera_pixel_equivalent), keeps it when it exists and is finite, and sums the kept ones in
// track order, so the mean is the reference's sequential sum divided by the count. The camera point
// is R (X - C) for the world-to-camera rotation R and the camera centre C of the pose (the reference
// holds t = -R C and evaluates R X + t; the two agree to rounding). Fewer than two kept residuals
// reject the landmark; a landmark that kept every supporting residual keeps its support; otherwise
// the support shrinks to the kept observations.
#include <cuda_runtime.h>

#include <string>
#include <vector>

#include "camera_models.cuh"
#include "gpu_solver.hpp"

namespace omvgba {

__global__ void __launch_bounds__(128)
    k_sfm_refresh(uint64_t landmarks, const double* __restrict__ rotation, const double* __restrict__ center,
                  const CameraDev* __restrict__ cameras, const double* __restrict__ points,
                  const uint8_t* __restrict__ active, const uint64_t* __restrict__ offset,
                  const uint32_t* __restrict__ track_pose, const uint32_t* __restrict__ track_intrinsic,
                  const double* __restrict__ track_pixel, const uint8_t* __restrict__ support_in,
                  uint8_t* __restrict__ support_out, uint8_t* __restrict__ update, double* __restrict__ error,
                  uint32_t* __restrict__ removed) {
  const uint64_t l = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (l >= landmarks) return;
  const uint64_t a = offset[l], b = offset[l + 1];
  removed[l] = 0;
  if (!active[l]) {
    update[l] = OMVGBA_REFRESH_SKIPPED;
    for (uint64_t o = a; o < b; ++o) support_out[o] = support_in[o];
    return;
  }
  const double X[3] = {points[3 * l], points[3 * l + 1], points[3 * l + 2]};
  double sum = 0.0;
  uint32_t kept = 0, supporting = 0;
  for (uint64_t o = a; o < b; ++o) {
    uint8_t keep = 0;
    if (support_in[o]) {
      ++supporting;
      const uint32_t p = track_pose[o];
      if (p != OMVGBA_NO_POSE) {
        const double* R = rotation + 9 * (size_t)p;
        const double* C = center + 3 * (size_t)p;
        const double d0 = X[0] - C[0], d1 = X[1] - C[1], d2 = X[2] - C[2];
        const double xc[3] = {R[0] * d0 + R[1] * d1 + R[2] * d2, R[3] * d0 + R[4] * d1 + R[5] * d2,
                              R[6] * d0 + R[7] * d1 + R[8] * d2};
        double r;
        if (camera_pixel_equivalent(cameras[track_intrinsic[o]], xc, track_pixel[2 * o], track_pixel[2 * o + 1], &r)) {
          sum += r;
          ++kept;
          keep = 1;
        }
      }
    }
    support_out[o] = keep;
  }
  if (kept < 2 || kept == supporting) {  // rejected or unchanged: the support stays as it was
    for (uint64_t o = a; o < b; ++o) support_out[o] = support_in[o];
    update[l] = kept < 2 ? OMVGBA_REFRESH_REJECTED : OMVGBA_REFRESH_UNCHANGED;
    if (kept >= 2) error[l] = sum / (double)kept;
    return;
  }
  update[l] = OMVGBA_REFRESH_PRUNED;
  error[l] = sum / (double)kept;
  removed[l] = supporting - kept;
}

namespace {

void check(cudaError_t e, const char* what) {
  if (e != cudaSuccess) throw SolveFailure{OMVGBA_CUDA_ERROR, std::string(what) + ": " + cudaGetErrorString(e)};
}

// Stream-ordered device buffer, freed on the stream when it goes out of scope.
struct StreamBuf {
  void* p = nullptr;
  cudaStream_t s;
  cudaMemPool_t pool;
  StreamBuf(cudaStream_t stream, cudaMemPool_t from) : s(stream), pool(from) {}
  StreamBuf(const StreamBuf&) = delete;
  StreamBuf& operator=(const StreamBuf&) = delete;
  ~StreamBuf() {
    if (p) cudaFreeAsync(p, s);
  }
  template <typename T>
  T* alloc(size_t count) {
    check(cudaMallocFromPoolAsync(&p, count ? sizeof(T) * count : 16, pool, s), "cudaMallocFromPoolAsync");
    return static_cast<T*>(p);
  }
};

}  // namespace

void gpu_sfm_refresh(Context* ctx, const SfmRefreshInput& in, SfmRefreshOutput& out) {
  check(cudaSetDevice(context_device(ctx)), "cudaSetDevice");
  cudaStream_t st = static_cast<cudaStream_t>(context_stream(ctx));
  const uint64_t L = in.landmark_count, N = in.track_count;
  std::vector<CameraDev> cams(in.intrinsic_count);
  const omvgba_intrinsic* intr = static_cast<const omvgba_intrinsic*>(in.intrinsics);
  for (uint64_t i = 0; i < in.intrinsic_count; ++i) cams[i] = make_camera_dev(intr[i]);
  cudaMemPool_t pool = static_cast<cudaMemPool_t>(context_pool(ctx));
  StreamBuf b_rot(st, pool), b_cen(st, pool), b_cam(st, pool), b_pts(st, pool), b_act(st, pool), b_off(st, pool),
      b_tp(st, pool), b_ti(st, pool), b_px(st, pool), b_sin(st, pool), b_sout(st, pool), b_upd(st, pool),
      b_err(st, pool), b_rem(st, pool);
  // All of the device memory before the first copy: a large copy waits for the stream, and at a wait the pool
  // gives back what it holds unused beyond its allowance. With the allocations between the copies every call
  // of 12M observations unmapped and mapped 150 MB again, and one in thirty stalled for 0.1 to 0.9 s in the
  // driver, on a call that takes 37 ms.
  double* rot = b_rot.alloc<double>(9 * in.pose_count);
  double* cen = b_cen.alloc<double>(3 * in.pose_count);
  CameraDev* dcam = b_cam.alloc<CameraDev>(cams.size());
  double* pts = b_pts.alloc<double>(3 * L);
  uint8_t* act = b_act.alloc<uint8_t>(L);
  uint64_t* off = b_off.alloc<uint64_t>(L + 1);
  uint32_t* tp = b_tp.alloc<uint32_t>(N);
  uint32_t* ti = b_ti.alloc<uint32_t>(N);
  double* px = b_px.alloc<double>(2 * N);
  uint8_t* sin_ = b_sin.alloc<uint8_t>(N);
  uint8_t* sout = b_sout.alloc<uint8_t>(N);
  uint8_t* upd = b_upd.alloc<uint8_t>(L);
  double* err = b_err.alloc<double>(L);
  uint32_t* rem = b_rem.alloc<uint32_t>(L);
  auto upload = [&](auto* to, const auto* from, size_t count) {
    check((cudaError_t)copy_to_device(to, from, sizeof(*to) * count, st), "upload");
  };
  upload(rot, in.rotation, 9 * in.pose_count);
  upload(cen, in.center, 3 * in.pose_count);
  upload(dcam, cams.data(), cams.size());
  upload(pts, in.points, 3 * L);
  upload(act, in.active, L);
  upload(off, in.track_offset, L + 1);
  upload(tp, in.track_pose, N);
  upload(ti, in.track_intrinsic, N);
  upload(px, in.track_pixel, 2 * N);
  upload(sin_, in.track_support, N);
  upload(err, out.reprojection_error, L);  // untouched entries come back as they were
  if (L > 0) {
    k_sfm_refresh<<<(unsigned)((L + 127) / 128), 128, 0, st>>>(L, rot, cen, dcam, pts, act, off, tp, ti, px, sin_,
                                                                 sout, upd, err, rem);
    check(cudaGetLastError(), "k_sfm_refresh launch");
  }
  std::vector<uint32_t> removed(L);
  check((cudaError_t)copy_from_device(out.track_support, sout, N, st), "download");
  check((cudaError_t)copy_from_device(out.landmark_update, upd, L, st), "download");
  check((cudaError_t)copy_from_device(out.reprojection_error, err, sizeof(double) * L, st), "download");
  check((cudaError_t)copy_from_device(removed.data(), rem, sizeof(uint32_t) * L, st), "download");
  check(cudaStreamSynchronize(st), "k_sfm_refresh");
  out.rejected_landmarks = 0;
  out.removed_observations = 0;
  for (uint64_t l = 0; l < L; ++l) {
    out.rejected_landmarks += out.landmark_update[l] == OMVGBA_REFRESH_REJECTED ? 1 : 0;
    out.removed_observations += removed[l];
  }
}

}  // namespace omvgba
