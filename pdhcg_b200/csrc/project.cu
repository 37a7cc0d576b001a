// project.cu -- cone projections of a vector (project.cuh) and their launchers.
#include "launch.cuh"
#include "project.cuh"

namespace pdhcg {

void launch_project_cones(int S, const ProjectArgs &a, cudaStream_t s)
{
    dispatch_s(S, [&](auto SC) {
        project_cones_kernel<SC.value><<<grid_for(a.ncones, WARPS), TPB, 0, s>>>(
            a.ncones, a.start, a.len, a.type, a.alpha, a.x, a.d, a.q, a.tau, a.psd_work, a.psd_off, a.fixed,
            a.cone_fixed, a.warm);
    });
}

void launch_project_sections(int S, const ProjectArgs &a, cudaStream_t s)
{
    dispatch_s(S, [&](auto SC) {
        project_sections_kernel<SC.value><<<grid_for(a.ncones, WARPS), TPB, 0, s>>>(
            a.ncones, a.start, a.len, a.type, a.alpha, a.x, a.d, a.q, a.tau, a.fixed, a.warm);
    });
}

} // namespace pdhcg
