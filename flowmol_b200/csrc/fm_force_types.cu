// fm_force_types.cu -- the list force kernel with Mie types and the Soddemann solvent.
#include <cuda_runtime.h>
#include <stdint.h>

#include "fm_force_list.cuh"

namespace fm {

template <int TPM>
static void launch_tpm(const FmDev &d, int record, int mode, cudaStream_t st)
{
    const int g = force_blocks(d.n, TPM);
#define FM_FORCE_CASE(R, M)                                                                     \
    if (record == R && mode == M) {                                                             \
        switch (d.precision + 2 * d.mie + 4 * d.solvent) {                                      \
        case 2: pdl_launch(k_force<TPM, R, M, 2>, g, FORCE_THREADS, st, d); break;              \
        case 3: pdl_launch(k_force<TPM, R, M, 3>, g, FORCE_THREADS, st, d); break;              \
        case 4: pdl_launch(k_force<TPM, R, M, 4>, g, FORCE_THREADS, st, d); break;              \
        case 5: pdl_launch(k_force<TPM, R, M, 5>, g, FORCE_THREADS, st, d); break;              \
        case 6: pdl_launch(k_force<TPM, R, M, 6>, g, FORCE_THREADS, st, d); break;              \
        default: pdl_launch(k_force<TPM, R, M, 7>, g, FORCE_THREADS, st, d); break;             \
        }                                                                                       \
        return;                                                                                 \
    }
    FM_FORCE_CASE(0, 0) FM_FORCE_CASE(0, 1) FM_FORCE_CASE(0, 2) FM_FORCE_CASE(0, 3)
    FM_FORCE_CASE(1, 0) FM_FORCE_CASE(1, 1) FM_FORCE_CASE(1, 2) FM_FORCE_CASE(1, 3)
#undef FM_FORCE_CASE
}

void launch_force_types(const FmDev &d, int record, int mode, int tpm, cudaStream_t st)
{
    switch (tpm) {
    case 1: launch_tpm<1>(d, record, mode, st); break;
    case 2: launch_tpm<2>(d, record, mode, st); break;
    case 4: launch_tpm<4>(d, record, mode, st); break;
    case 16: launch_tpm<16>(d, record, mode, st); break;
    default: launch_tpm<8>(d, record, mode, st); break;
    }
}

}  // namespace fm
