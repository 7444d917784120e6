// Host-side view of the LayerNorm backward's geometry rule (ln_geometry.h is what the launch code
// runs), for the CPU tests; no CUDA involved.
#include "../ln_geometry.h"

// out: vectors per lane, warps per row, rows of a CTA.  Returns 0, or -1 where no geometry exists.
extern "C" int tp_ln_bwd_geometry(int H, int rows, int sms, int* out) {
  if (rows <= 0 || !tp::ln_bwd_geometry(H, rows, sms, &out[0], &out[1])) return -1;
  out[2] = tp::ln_bwd_rows(out[0], out[1]);
  return 0;
}
