// Programmatic dependent launch of a chain of kernels on one stream, for the slice loop of the plasma march.
//
// A kernel launched with launch_pdl may start while the kernel before it on the stream still runs, once every CTA of that
// one has called pdl_next() or ended. Its code up to pdl_wait() overlaps the kernel before it; pdl_wait() returns when that
// kernel has ended and its stores are visible. In the chain every kernel calls pdl_wait() and only then pdl_next(): so when
// a kernel starts early, the kernel before it is past its own wait, i.e. everything up to the kernel before that one is
// complete. Before its wait a kernel may therefore read what the kernel directly before it does not write, and
// writes nothing. Without the launch attribute both calls do nothing.
//
// What the kernel directly before writes is not constant for the life of the kernel that reads it: that one is resident
// already. So such memory is never read through `const __restrict__` pointers or __ldg, which promise that it is and let the
// compiler take a non-coherent load or move the load above the wait. A kernel takes it as Handed<T> (or inside its argument
// struct, or as a plain T*) and reads it by ordinary loads after pdl_wait(), which the clobber holds there. Tables and what
// was written two or more kernels earlier may be read as constant.
#pragma once
#include "g3d_common.cuh"

namespace g3d {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// memory handed over by the kernel before: a pointer without aliasing promises, whose values are read after pdl_wait()
template <class T>
struct Handed {
    const T* p;
    __device__ __forceinline__ T operator[](long i) const { return p[i]; }
};

template <class... P, class... A>
void launch_pdl(cudaStream_t s, void (*kern)(P...), dim3 grid, dim3 block, size_t smem, A&&... args) {
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = s;
    cfg.attrs = at; cfg.numAttrs = 1;
    G3D_CUDA(cudaLaunchKernelEx(&cfg, kern, P(args)...));
}

}  // namespace g3d
