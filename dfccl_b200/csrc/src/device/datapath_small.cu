// The bodies of small reductions (datapath.h: reduceSmall), compiled for few registers.
#define DF_DATAPATH_SMALL_IMPL
#include "datapath.h"
