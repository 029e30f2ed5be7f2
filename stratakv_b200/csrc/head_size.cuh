// What the attention files, which are built once per head size, have besides common.cuh: the head size.
#pragma once

#include "common.cuh"

#ifndef SKV_HEAD_DIM
#error "compile with -DSKV_HEAD_DIM=<head size, a multiple of 16>"
#endif
