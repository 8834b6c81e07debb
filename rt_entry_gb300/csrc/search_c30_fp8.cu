// Instantiations of search_kernel for d <= 960, FP8-E4M3.
#define SEARCH_C 30
#define SEARCH_PREC kPrecFP8
#define SEARCH_FN search_lookup_c30_fp8
#define SEARCH_CASES RTE_CASE(0, 2) RTE_CASE(1, 2) RTE_CASE(2, 2) RTE_CASE(4, 2) RTE_CASE(8, 2) RTE_CASE(4, 4) RTE_CASE(8, 4) RTE_CASE(4, 8) RTE_CASE(8, 8)
#include "search_inst.inc"
