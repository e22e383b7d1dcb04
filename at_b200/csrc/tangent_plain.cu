/* Tangent kernel of the lattices with hand-written element derivatives, in the
 * "exact" arithmetic (compiled with -fmad=false like track_exact.cu, so the
 * tracked values equal those of the exact tracking kernel; the derivatives use
 * explicit fma()). */
#define ATB_FAST 0
#define ATB_NO_TRACK_KERNEL
#include "tangent_plain.cuh"
