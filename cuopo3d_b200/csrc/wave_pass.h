// Interface of the plane-wave solver's whole-crystal kernel (wave_pass.cu).
#pragma once

#include "opo_internal.h"

namespace opo {

template <typename C> struct WaveArgs {
    TPassArgs<C> rk;      // fields, pump source and coupled-wave constants (its plan is unused)
    unsigned M, bw, K;    // block length n / K, samples per row M / K, cluster size
    int nsample;          // plan stages on the sample buffer (their radices' product is K)
    unsigned xregion;     // values per field of the sample buffer
    AxisPlan plan;
    TileGeom g;           // block buffer: one line of M values per field
    const C *tw;
    const C *tab[2][3];   // phase tables: crystal step, closing pass
    const C *eom;         // closing pass, or null
    const C *ph_steps;    // exp(i dk z) per t-pass, [tp][2][3] (rk.use_phase)
    int n_steps;
    unsigned mask;        // fields transformed by a step
    int closing;          // the closing pass is a round trip's (EOM, GDD and mirrors)
    unsigned close_mask;
};

template <typename C> cudaError_t configure_wave_kernels();
// Whether a cluster of K CTAs with smem bytes each can be resident.
template <typename C> bool wave_fits(int K, size_t smem);
template <typename C> cudaError_t launch_wave(const WaveArgs<C> &w, size_t smem, cudaStream_t st);

}  // namespace opo
