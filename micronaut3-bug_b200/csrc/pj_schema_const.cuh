/*
 * pj_schema_const.cuh — the model tables in constant memory: one copy per translation unit, which sets its own.
 */
#ifndef PJ_SCHEMA_CONST_CUH
#define PJ_SCHEMA_CONST_CUH
#include "pj_core.cuh"
namespace pj { static __constant__ Schema c_schema; }
#endif
