// cov_prep.h -- sequence weights and the gap filter on the device (internal).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace covgpu {

// unnormalised position-based weights w[N] of the alignment ax [N][Lp]
// (inv is scratch [L][4])
cudaError_t launch_weights_pb(const uint8_t* ax, int N, int L, int Lp, double* inv, double* w, cudaStream_t st);
// unnormalised GSC weights w[N] (scratch of gsc_scratch_bytes(N, L) bytes,
// 16-byte aligned)
size_t      gsc_scratch_bytes(int N, int L);
int         gsc_max_sequences();   // of the current device: 16384, 8192 without clusters of 16 CTAs (0: error)
cudaError_t launch_weights_gsc(const uint8_t* ax, int N, int L, int Lp, void* scratch, double* w, cudaStream_t st);
// useme[L]: 1 where the weighted residue fraction is at least 1 - gapthresh
// (wgt null: unit weights)
cudaError_t launch_gapfilter(const uint8_t* ax, const double* wgt, int N, int L, int Lp, double gapthresh, int* useme,
                             cudaStream_t st);

// rows of L bytes (src: 256-byte aligned, 20 bytes of slack) to a pitch of Lp
cudaError_t launch_spread_rows(const uint8_t* src, int N, int L, int Lp, uint8_t* dst, cudaStream_t st);

}  // namespace covgpu
