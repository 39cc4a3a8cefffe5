// The source model's panel images: the emission profile and the beam filter's thickness, read at panel coordinates.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace citrus {

// Emission profile, off-focal table and beam filter of the source (all optional; float64 tables on the device).
struct SourceExtras {
  const double* profile;    // [rows, channels] relative emission toward each pixel centre, or null
  const double* thickness;  // [t_rows, channels] filter thickness in cm at the pixel centres, or null
  int t_rows;
  const double* off_nodes;  // [n_off] ascending distances past the field edge in cm, or null
  const double* off_values; // [n_off] emission there relative to the field edge
  int n_off;
  int rows, channels;
  double d_row, d_ch, off_row, off_ch;
  double filter_density;
};

// Bilinear at panel coordinates, held at the outermost pixel centres (source.py:484-510)
__device__ inline double panel_interpolate(const double* __restrict__ img, int img_rows, const SourceExtras& ex,
                                           double u, double v) {
  const double xc = fmin(fmax((u + ex.off_ch) / ex.d_ch + (ex.channels - 1) * 0.5, 0.0), ex.channels - 1.0);
  const double xr = fmin(fmax((v + ex.off_row) / ex.d_row + (ex.rows - 1) * 0.5, 0.0), ex.rows - 1.0);
  const int c0 = min(max((int)floor(xc), 0), max(ex.channels - 2, 0)), c1 = min(c0 + 1, ex.channels - 1);
  int r0 = min(max((int)floor(xr), 0), max(ex.rows - 2, 0)), r1 = min(r0 + 1, ex.rows - 1);
  if (img_rows == 1) r0 = r1 = 0;
  const double wc = fmin(fmax(xc - c0, 0.0), 1.0), wr = fmin(fmax(xr - r0, 0.0), 1.0);
  const double* a = img + (int64_t)r0 * ex.channels;
  const double* b = img + (int64_t)r1 * ex.channels;
  const double top = a[c0] + (a[c1] - a[c0]) * wc;
  const double bottom = b[c0] + (b[c1] - b[c0]) * wc;
  return top + (bottom - top) * wr;
}

}  // namespace citrus
