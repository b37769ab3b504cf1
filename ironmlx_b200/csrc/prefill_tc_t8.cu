#include "prefill_tc.cuh"

namespace imx::prefill {
IMX_TC_FORMAT(FMT_T8)
}
