// The host build of sc_ddmath.cuh for ddmath_device_check.cu (in a file that
// nvcc compiles, the tables are on the device only).
#include "sc_ddmath.cuh"

extern "C" void host_eval(double x, double y, double* log_cr, double* atan_cr, double* log_quick) {
    *log_cr = sc::ddm::log_dd(x);
    *atan_cr = sc::ddm::atan_dd(y);
    *log_quick = sc::ddm::log_fast(x);
}
