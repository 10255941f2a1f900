// 2D row passes (double) with double potential products: complex time steps.
#define QSG_DOUBLE_UNIT 1
#include "qsg_row_f64.cu"
