// Stepper instantiation for dimension SPD_D and degree SPD_P, both given on
// the compiler's command line (one translation unit each: spd_gb300/build.py).
#include "spd_stepper.cuh"

namespace spd_host {
template StepperBase* make_stepper_of<SPD_D, SPD_P>();
}  // namespace spd_host
