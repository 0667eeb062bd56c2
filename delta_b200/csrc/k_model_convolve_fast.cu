// The model convolve for n_max = 6, and the choice of the instantiation
// (model_convolve_fast.cuh).
#include "model_convolve_fast.cuh"

namespace dgpu {

extern template bool launch_model_convolve_nx<3>(cudaStream_t, const SubtractArgs&, const int2*, int, size_t);
extern template bool launch_model_convolve_nx<4>(cudaStream_t, const SubtractArgs&, const int2*, int, size_t);
extern template bool launch_model_convolve_nx<5>(cudaStream_t, const SubtractArgs&, const int2*, int, size_t);
extern template bool launch_model_convolve_nx<6>(cudaStream_t, const SubtractArgs&, const int2*, int, size_t);

size_t model_convolve_fast_smem(int nx, int ks, int TH, const DevFields& F) {
  const int kh = (ks - 1) / 2;
  const int nrows = TH + 2 * kh;
  const int kb = (ks + 7) / 8;
  return sizeof(float) * (2 * static_cast<size_t>((nrows + 1) / 2) * fast_rw(ks) +
                          static_cast<size_t>(nx) * (nrows + kFPad) * kFTW + static_cast<size_t>(nx) * 3 * 8 * kb +
                          static_cast<size_t>(nx) * (nx + 1) +
                          static_cast<size_t>(lattice_cap(F, TH)));
}

bool model_convolve_fast_available(int nx, int ks) {
  const int kb = (ks + 7) / 8;
  return (nx == 3 || nx == 4 || nx == 5 || nx == 6 || nx == 7) && kb >= 2 && kb <= 5;
}

bool launch_model_convolve_fast(cudaStream_t s, const SubtractArgs& a, const int2* orders, int TH) {
  const int nx = a.n_max + 1;
  if (!model_convolve_fast_available(nx, a.ks)) return false;
  const size_t smem = model_convolve_fast_smem(nx, a.ks, TH, a.F);
  switch (nx) {
    case 3: return launch_model_convolve_nx<3>(s, a, orders, TH, smem);
    case 4: return launch_model_convolve_nx<4>(s, a, orders, TH, smem);
    case 5: return launch_model_convolve_nx<5>(s, a, orders, TH, smem);
    case 6: return launch_model_convolve_nx<6>(s, a, orders, TH, smem);
    case 7: return launch_model_convolve_nx<7>(s, a, orders, TH, smem);
    default: return false;
  }
}

}  // namespace dgpu
