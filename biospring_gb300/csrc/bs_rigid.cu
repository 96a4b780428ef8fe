// bs_rigid.cu -- rigid-body dynamics of the step (RigidBodiesManager::SolveRigidBodiesDynamic,
// src/rigidbody/RigidBodiesManager.cpp:45-60).
//
// The step kernel leaves the total force of every rigid particle (springs to non-rigid partners,
// nonbonded terms, viscosity, IMPALA, external force) in rforce and does not move it. Then one
// block per body:
//   1. sums the force and the torque (x_i - X) x f_i over the body's members
//      (RigidBody::computeParticleForceAndTorque, RigidBody.cpp:567-580) in float-float;
//   2. advances the body (RigidBody::solve, RigidBody.cpp:455-483): a = F / M, v += a dt,
//      X += v dt + a/2 dt^2, L += tau dt, omega = I^-1 L with the sphere inertia I = 2/5 M,
//      rotation by the quaternion (omega sin(|omega| dt / 2), cos(|omega| dt / 2)) (the axis is
//      omega itself, not normalised, as in the reference), renormalised;
//   3. places every member at X + q p0 q^-1 with velocity (new - old) / dt
//      (RigidBody::integrateParticleVelocity, RigidBody.cpp:600-635), p0 being the member's
//      offset from the barycentre at set-up, taken by its index within its own body.
// Float operations are written without contraction, in the reference's order, so a body
// follows the reference up to the order of the force sum.

#include "bs_rigid.cuh"

namespace bsg
{
namespace
{

__global__ void __launch_bounds__(kRigidBlock) k_rigid(Params p)
{
    Ctl *ctl = p.ctl;
    // the step kernel advances ctl->steps when it completes a step; bodies that already moved
    // for this step count (a status bit stopped the step kernel) stay
    const long long steps = *(volatile const long long *)&ctl->steps;
    if (steps == *(volatile const long long *)&ctl->rigid_steps)
        return;
    const int pend = rigid_body_step(p, blockIdx.x, ctl->sbuf ^ 1);
    // raised bits stop the next kernels
    if (pend)
        atomicOr(&ctl->status, pend);
    // the last block records the step as done: every block has passed its check by then
    __syncthreads();
    __shared__ bool last;
    if (threadIdx.x == 0)
    {
        __threadfence();
        last = atomicAdd(&ctl->done_rigid, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (last && threadIdx.x == 0)
    {
        ctl->rigid_steps = steps;
        ctl->done_rigid = 0u;
    }
}

} // namespace

int launch_rigid(const Params &p, cudaStream_t st)
{
    k_rigid<<<p.nbody, kRigidBlock, 0, st>>>(p);
    return 1;
}

} // namespace bsg
