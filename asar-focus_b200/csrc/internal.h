// Host-side helpers shared by the planner (host.cpp) and the per-stage entry points (stages.cpp).
#pragma once

#include <complex>
#include <vector>

#include "asarf.h"
#include "fft.cuh"
#include "params.h"

namespace asarf {

// FFT schedule of one length with its digit-reversal map and FP64-computed twiddles.
struct HostFft {
    FftPlan plan{};
    std::vector<int> drev;
    std::vector<float2> tw;
};

bool smooth(int n);
// Longest synthetic aperture in lines over the range swath (CalcAperturePixels).
int max_aperture_pixels(const asarf_scene& s);
// Ground-to-slant SRGR polynomial (5 coefficients) and ground sample count for a multilooked
// block of azimuth_size lines at line interval lti (SlantRangeToGroundRangeInterpolation setup).
int srgr_poly(const asarf_scene& s, double slant_first, int range_size, int azimuth_size, double lti, double poly[5],
              int* ng);
bool build_fft(int n, HostFft& h);
// Same with an explicit radix sequence (product n), e.g. a compile-time schedule's; without the
// twiddle table where only the schedule and order are wanted.
bool build_fft_radices(int n, const std::vector<int>& radices, HostFft& h, bool with_twiddles = true);
// Radices of the strided azimuth pass (at most 9) and of the contiguous one (at most 8): the compiled schedule
// of that length when there is one (the run-time loops take 9 to 25 % and 10 % longer, more than a
// smaller sum of radices gives), else two or three factors, nearest to each other and largest first;
// lengths that have none take their prime factors.
std::vector<int> strided_radices(int n);
std::vector<int> block_radices(int n);
// Contiguous length n2 of the azimuth split N = n1 * n2 for nk columns (halo hl, hr of the
// range-Doppler tile).
int choose_az_n2(int N, int nk, int hl, int hr, bool absolute_phase);
// Mean gain error of a transform with this schedule: its float twiddles (from the table at every power,
// or by recurrence) and radix constants are rounded, which scales all outputs alike by some 1e-8 to
// 1e-7; its inverse has the same.
double transform_gain(const HostFft& h, bool table_powers);
// 1 / N of the azimuth transforms with `gain`, the sum of those of the two forward and two inverse passes, taken
// back: it is the one error of theirs that all samples share.
inline float azimuth_scale(int N, double gain) { return static_cast<float>(1.0 / (N * (1.0 + gain))); }
int largest_divisor_le(int n, int cap);
// Rows of a TMA box of the range-Doppler tile (n2 rows of wt complex values): all n2 up to 256, else their
// largest divisor whose boxes each start on a 128-byte boundary of shared memory, as a tensor copy must;
// 0 where none does (n2 = 343, odd rows: the tile then arrives by plain loads).  The strided pass's
// rows are whole multiples of 128 bytes.
int rd_box_rows(int n2, int wt);
// TMA maps (128-byte blobs) of the azimuth passes over an image pair a, b of n1 * n2 rows of `pitch`
// complex values, nk of them data: strided views of a and b (nb tiles of xt columns, n1_box of the
// n1 rows a box) and the contiguous view of a (wt columns, n2_box rows).
bool make_azimuth_maps(float2* a, float2* b, int nk, long long pitch, int n1, int n2, int xt, int nb, int n1_box, int wt,
                       int n2_box, void* map_a3, void* map_b3, void* map_a2);
int choose_rc_len(int nr);
int32_t fft_size_above(int32_t v);
// Device tables of a range transform: the matched filter (fft.plan.n entries) from a replica of nc
// samples in device memory, and the twiddle tables of a compile-time length.
MatchedFilterArgs matched_filter_args(const float2* d_chirp, int nc, const HostFft& fft, float2* d_mf);
TwiddleArgs ct_twiddle_args(int L, float2* d_out);

}  // namespace asarf
