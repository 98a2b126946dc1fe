// The kernels of a decode step's few rows, for the building-block library.
#include "linear_rows_body.cuh"
#include "token_rows_body.cuh"
