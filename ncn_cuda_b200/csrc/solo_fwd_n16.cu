#define NCN_NG 16
#include "solo_inst.cuh"
