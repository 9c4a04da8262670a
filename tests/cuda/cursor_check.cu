// cursor_check.cu - host build of the rule for the ray queue's 32-bit cursor.
#include "../../risltc_gb300/csrc/cuda/ris_wavefront.cuh"

extern "C" int risltc_test_cursor_holds(unsigned rays, unsigned threads) {
	return risltc::cursor_holds(rays, threads) ? 1 : 0;
}
