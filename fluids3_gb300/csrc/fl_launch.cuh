// Launches that begin before the one before them is complete (programmatic
// dependent launch). Included inside each file's anonymous namespace.
#pragma once

// The first statement of every kernel that launch() starts: waits until the
// launch before it is complete and its writes are visible (at once if its
// launch waited for that already). What the launch before it wrote changes
// during such a kernel's own lifetime, so its parameters are not __restrict__
// (const with it promises that they do not change in that time, and lets the
// compiler read them before the wait, or past the coherent path), nor are they
// read through the non-coherent path by hand. The functions that a kernel calls
// after the wait may have such parameters: the promise then begins there.
// Nothing lets a launch begin earlier than when the blocks of the one before it
// have ended: blocks that waited beside running ones were packed onto the
// multiprocessors that those left free (100,000 points at the default
// settings, one step: 115 us with such early starts, 76 without, 83 with
// ordinary launches).
__device__ __forceinline__ void follow_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// A pointer whose loads cannot come before follow_previous, for the loads that
// the compiler could otherwise move across it.
template <class T>
__device__ __forceinline__ T *after_wait(T *p) {
    asm volatile("" : "+l"(p));
    return p;
}

// A launch that may begin before the one before it in the stream is complete
// (its kernel calls follow_previous first): the gap between the two is shorter.
// Gradients of 10 steps of 65,536 points, about 400 launches: 4,149 us with
// ordinary launches, 3,356 with these; a step of 2,048 points, 10 launches: 37.9
// and 35.9.
template <class... P, class... A>
inline void launch(void (*kernel)(P...), dim3 grid, int block, size_t smem, cudaStream_t stream, A &&...args) {
    cudaLaunchAttribute early = {};
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c = {};
    c.gridDim = grid;
    c.blockDim = dim3((unsigned)block);
    c.dynamicSmemBytes = smem;
    c.stream = stream;
    c.attrs = &early;
    c.numAttrs = 1;
    (void)cudaLaunchKernelEx(&c, kernel, static_cast<A &&>(args)...);   // (the caller checks for errors)
}
