// Instantiations of the convolution column pass: masked problems.
#include "sc_inst_colc.cuh"

ColFn sc_colc_fn_full(int kr, int n, int L) { return colc_table<CONV_FULL>(kr, n, L); }
