// staged_plain.cuh - the plain FP64 engines' frames as a pipeline of stages.
//
// The same per-pixel work as plain_kernel (plain_kernel.cuh), operation for
// operation, split so that no lane waits for another kind of work.  One thread
// per pixel left 13 to 18 of 32 lanes active (a warp ran its longest orbit in
// every estimate, its longest march in every ray, and its AO rays one after
// the other), and the slowest warp's chain of march, normals, shadow and AO
// rays set the frame's time.  What bounds the stages now is FP64 latency and
// issue, and in stages P and S the longest single ray.  One thread per pixel
// -> stages: Mandelbox 801x451, 4 AO rays, 2.33 -> 1.56 ms of kernels; a
// pseudo-Kleinian view 320x240, 4 AO rays, 33.7 -> 6.8 ms.
