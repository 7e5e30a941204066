// Host build of the server's memory estimate (csrc/footprint.h).
#include "../../collisiondetection_gb300/csrc/footprint.h"

extern "C" int64_t hc_footprint(int64_t nfaces, int64_t nverts) { return ccd::request_footprint(nfaces, nverts); }
