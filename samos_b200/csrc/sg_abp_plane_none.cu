// Step-kernel variants of the active-Brownian program: plane, no aligner.
#include "sg_abp_launch.cuh"

void sg::launch_abp_plane_none(const AbpLaunch& L) { launch_abp_unit<HOT_PLANE, ABP_ALIGN_NONE>(L); }
