// One part of the engine's kernel instantiations (LUMEN_PART, 0 .. LUMEN_N_PARTS - 1), compiled in parallel with
// the others; lumen_b200.cu declares each launcher extern.
#ifndef LUMEN_PART
#error "compile with -DLUMEN_PART=k"
#endif
// the wavefront's step with tangents calls the elementary functions: its code is the longest of the kernels, and inlined
// they cost it more instruction fetch than the calls (ground-wall tank with four tangents, 2,000,000 photons: 11.3 ->
// 10.4 ms, the track events 13.3 -> 13.1); the other kernels lose 1 to 2 % with them called
#if LUMEN_PART >= 17
#define L_MATH static __device__ __noinline__
#endif
#include "engine.cuh"

#define LUMEN_INST_SHAPE(G, B, M, T, A, N) template LUMEN_SHAPE_DECL(G, B, M, T, A, N)
#define LUMEN_INST_QUERY(T, N) template LUMEN_WAVE_QUERY_DECL(T, N)
#define LUMEN_INST_STEP(G, B, E, N) template LUMEN_WAVE_STEP_DECL(G, B, E, N)
#if LUMEN_PART == 0
LUMEN_SHAPES_0(LUMEN_INST_SHAPE)
#elif LUMEN_PART == 1
LUMEN_SHAPES_1(LUMEN_INST_SHAPE)
#elif LUMEN_PART == 2
LUMEN_SHAPES_2(LUMEN_INST_SHAPE)
#elif LUMEN_PART == 3
LUMEN_SHAPES_3(LUMEN_INST_SHAPE)
#elif LUMEN_PART == 4
LUMEN_SHAPES_4(LUMEN_INST_SHAPE)
#elif LUMEN_PART == 5
LUMEN_SHAPES_5(LUMEN_INST_SHAPE)
#elif LUMEN_PART == 6
LUMEN_SHAPES_6(LUMEN_INST_SHAPE)
#elif LUMEN_PART == 7
LUMEN_SHAPES_7(LUMEN_INST_SHAPE)
#elif LUMEN_PART == 8
LUMEN_SHAPES_8(LUMEN_INST_SHAPE)
#elif LUMEN_PART == 9
LUMEN_SHAPES_9(LUMEN_INST_SHAPE)
#elif LUMEN_PART == 10
#define LUMEN_INST_FILL(E, N) template LUMEN_WAVE_FILL_DECL(E, N)
LUMEN_WAVE_FILLS(LUMEN_INST_FILL)
LUMEN_WAVE_QUERIES_10(LUMEN_INST_QUERY)
#elif LUMEN_PART == 12
LUMEN_WAVE_QUERIES_12(LUMEN_INST_QUERY)
#elif LUMEN_PART == 13
LUMEN_WAVE_QUERIES_13(LUMEN_INST_QUERY)
#elif LUMEN_PART == 14
LUMEN_WAVE_STEPS_14(LUMEN_INST_STEP)
#elif LUMEN_PART == 15
LUMEN_WAVE_STEPS_15(LUMEN_INST_STEP)
#elif LUMEN_PART == 16
LUMEN_WAVE_STEPS_16(LUMEN_INST_STEP)
#elif LUMEN_PART == 17
LUMEN_WAVE_STEPS_17(LUMEN_INST_STEP)
#elif LUMEN_PART == 18
LUMEN_WAVE_STEPS_18(LUMEN_INST_STEP)
#elif LUMEN_PART == 19
LUMEN_WAVE_STEPS_19(LUMEN_INST_STEP)
#elif LUMEN_PART == 20
LUMEN_WAVE_STEPS_20(LUMEN_INST_STEP)
#elif LUMEN_PART == 11
template int launch_event_locate<0>(const DScene&, const LumenSource&, int32_t*, cudaStream_t);
template int launch_event_locate<1>(const DScene&, const LumenSource&, int32_t*, cudaStream_t);
template int launch_photons<0>(const Launch&, int32_t*, float*, cudaStream_t);
template int launch_photons<1>(const Launch&, int32_t*, float*, cudaStream_t);
template int launch_query<float>(const DScene&, const float*, const int32_t*, const int32_t*, float, int64_t, int32_t*,
                                 float*, cudaStream_t);
template int launch_query<double>(const DScene&, const double*, const int32_t*, const int32_t*, double, int64_t,
                                  int32_t*, double*, cudaStream_t);
template int launch_locate<float>(const DScene&, const float*, int64_t, int32_t*, cudaStream_t);
template int launch_locate<double>(const DScene&, const double*, int64_t, int32_t*, cudaStream_t);
#endif
