// One velocity-Verlet step around an evaluation, in two kernels.
#pragma once

#include <cuda_runtime.h>

namespace sxb {

// The step moves 15 doubles per atom (260 KB for 2,160 atoms: far below a microsecond of HBM time); what it costs is
// launches and waits.  As tensor expressions it took 17 launches and, with each result read by its own copy, two waits besides
// that of the evaluation; here each half is one launch whose last block writes the one number that the host decides or reports
// by into mapped memory: a step of 2,160 atoms went from 1,451 to 1,283 us, its neighbor lists included.
// The operations and their rounding are those of the expressions  v += half * f / m;  x += dt * v  one by one (no FMA),
// so a trajectory does not depend on which of the two forms ran.
constexpr int kMdThreads = 128;
constexpr int kMdBlocks = 592;       // four per SM; a larger system strides

struct MdWorkspace {
    unsigned long long largest;      // bits of a non-negative double: ordered like the number, a NaN above all
    unsigned int arrived;            // blocks that have left their part; the last one puts both back to zero
    unsigned int pad;
    double partial[kMdBlocks];
};

// First half: kick, drift, and the largest squared displacement from the positions of the neighbor list.
__global__ void __launch_bounds__(kMdThreads) md_advance_kernel(int n, double dt, double half, double* __restrict__ x,
                                                                double* __restrict__ v, const double* __restrict__ f,
                                                                const double* __restrict__ m, const double* __restrict__ x_ref,
                                                                MdWorkspace* __restrict__ ws, double* __restrict__ host)
{
    __shared__ unsigned long long block_max;
    if (threadIdx.x == 0) block_max = 0;
    __syncthreads();
    unsigned long long largest = 0;
    for (int i = blockIdx.x * kMdThreads + threadIdx.x; i < n; i += gridDim.x * kMdThreads) {
        const double mass = m[i];
        double moved = 0.0;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const long j = 3l * i + q;
            const double vel = __dadd_rn(v[j], __ddiv_rn(__dmul_rn(half, f[j]), mass));
            const double pos = __dadd_rn(x[j], __dmul_rn(dt, vel));
            v[j] = vel;
            x[j] = pos;
            const double d = __dadd_rn(pos, -x_ref[j]);
            moved = __dadd_rn(moved, __dmul_rn(d, d));
        }
        const unsigned long long bits = static_cast<unsigned long long>(__double_as_longlong(moved)) & 0x7fffffffffffffffull;
        largest = bits > largest ? bits : largest;
    }
    if (largest != 0) atomicMax(&block_max, largest);
    __syncthreads();
    if (threadIdx.x != 0) return;
    atomicMax(&ws->largest, block_max);
    __threadfence();
    if (atomicAdd(&ws->arrived, 1u) + 1u != gridDim.x) return;
    __threadfence();
    host[0] = __longlong_as_double(static_cast<long long>(atomicExch(&ws->largest, 0ull)));
    ws->arrived = 0;
}

// Second half: the forces leave the evaluator's buffer, the second kick, and sum(m v^2) in a fixed order.
__global__ void __launch_bounds__(kMdThreads) md_finish_kernel(int n, double half, double* __restrict__ v,
                                                               const double* __restrict__ m, const double* __restrict__ forces,
                                                               double* __restrict__ f_out, MdWorkspace* __restrict__ ws,
                                                               double* __restrict__ host)
{
    __shared__ double part[kMdThreads];
    __shared__ bool last;
    double sum = 0.0;
    for (int i = blockIdx.x * kMdThreads + threadIdx.x; i < n; i += gridDim.x * kMdThreads) {
        const double mass = m[i];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const long j = 3l * i + q;
            const double force = forces[j];
            f_out[j] = force;
            const double vel = __dadd_rn(v[j], __ddiv_rn(__dmul_rn(half, force), mass));
            v[j] = vel;
            sum += mass * vel * vel;
        }
    }
    const auto reduce = [&](double value) {
        part[threadIdx.x] = value;
        __syncthreads();
        for (int width = kMdThreads / 2; width > 0; width >>= 1) {
            if (threadIdx.x < width) part[threadIdx.x] += part[threadIdx.x + width];
            __syncthreads();
        }
        return part[0];
    };
    const double block_sum = reduce(sum);
    if (threadIdx.x == 0) {
        ws->partial[blockIdx.x] = block_sum;
        __threadfence();
        last = atomicAdd(&ws->arrived, 1u) + 1u == gridDim.x;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double total = 0.0;
    for (int b = threadIdx.x; b < gridDim.x; b += kMdThreads) total += __ldcg(&ws->partial[b]);
    total = reduce(total);
    if (threadIdx.x == 0) {
        host[0] = total;
        ws->arrived = 0;
    }
}

}  // namespace sxb
