#define NCN_NG 8
#include "solo_inst.cuh"
