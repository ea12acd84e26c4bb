// Device functions and launchers of libhpgpu that no public entry point reaches by themselves, as C functions on host
// arrays for the tests (device_checks.py compiles and links this against the library).
#include "hp_internal.cuh"

extern "C" {

int dc_solve_capacity() { return hp::mbis_solve_capacity(); }

}  // extern "C"
