/* temporally blocked pass of small elastic grids for FDORDER=8 */
#include "dsh_tb.h"

namespace dsh {
template <bool P2, int MAXT>
static TbFn tb_pick(int mode)
{
    return mode == TB_ADJ     ? tb_pass<8, P2, TB_ADJ, MAXT>
           : mode == TB_STORE ? tb_pass<8, P2, TB_STORE, MAXT>
                              : tb_pass<8, P2, TB_FWD, MAXT>;
}
template <int MAXT>
static TbFn tb_p2(int mode, bool p2)
{
    return p2 ? tb_pick<true, MAXT>(mode) : tb_pick<false, MAXT>(mode);
}
TbFn tb_kernel_fd8(int mode, bool p2, int nthr)
{
    return nthr <= TB_FEW_THREADS   ? tb_p2<TB_FEW_THREADS>(mode, p2)
           : nthr <= TB_MID_THREADS ? tb_p2<TB_MID_THREADS>(mode, p2)
                                    : tb_p2<TB_MAX_THREADS>(mode, p2);
}
}  // namespace dsh
