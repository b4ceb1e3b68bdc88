// stream_kernels.cu -- the STREAM kernels (stream.cuh) of the extents the
// configurations name, several variants each for the tuner to choose from.
//
// Two stages and small items, with as many CTAs an SM as shared memory holds,
// beat deep rings of large items where lines are short (96 MB, before / with the
// variant added): 8^3 c64 45.0 / 37.2 us, 8x8x16 c128 45.4 / 38.4 and c64 45.2 /
// 38.3, 16^3 c64 40.6 / 36.9; 24^3 and 23^3 c64, one volume
// a stage on a thread a line, beat VOLUME (72.8 / 58.1 and 95.0 / 80.5 us).
#include "stream.cuh"

namespace fft3d {

void register_stream_kernels(std::vector<KernelEntry> &out)
{
    // complex double (ring must fit 227 KB per CTA, MINB CTAs per SM)
    FFT3D_STREAM(6, 6, 6, double, 0, 8, 288, 3, 1);
    FFT3D_STREAM(6, 6, 6, double, 0, 16, 576, 2, 1);
    FFT3D_STREAM(8, 8, 8, double, 0, 4, 256, 4, 1);
    FFT3D_STREAM(8, 8, 8, double, 0, 2, 128, 3, 2);
    FFT3D_STREAM(8, 8, 8, double, 0, 8, 512, 2, 1);
    FFT3D_STREAM(8, 8, 8, double, 0, 1, 64, 3, 8);   // one volume per item: even tails
    FFT3D_STREAM(8, 8, 8, double, 0, 1, 64, 4, 6);
    FFT3D_STREAM_BST(8, 8, 8, double, 0, 1, 64, 4, 6);
    FFT3D_STREAM(12, 12, 12, double, 0, 2, 288, 2, 1);
    FFT3D_STREAM(12, 12, 12, double, 0, 1, 160, 3, 2);
    FFT3D_STREAM(16, 16, 16, double, 0, 1, 256, 2, 1);
    FFT3D_STREAM(16, 16, 16, double, 0, 1, 256, 3, 1);
    FFT3D_STREAM_BST(16, 16, 16, double, 0, 1, 256, 3, 1);
    FFT3D_STREAM(17, 17, 17, double, 0, 1, 320, 2, 1);
    FFT3D_STREAM(17, 17, 17, double, 1, 1, 320, 2, 1);
    FFT3D_STREAM(17, 17, 17, double, 0, 1, 320, 1, 2);
    FFT3D_STREAM_BST(17, 17, 17, double, 0, 1, 320, 2, 1);
    FFT3D_STREAM_BST(17, 17, 17, double, 2, 1, 320, 2, 1);  // CRT cosine half
    FFT3D_STREAM(8, 8, 16, double, 0, 4, 512, 2, 1);
    FFT3D_STREAM(8, 8, 16, double, 0, 2, 256, 4, 1);
    FFT3D_STREAM(13, 13, 13, double, 0, 1, 192, 3, 2);
    FFT3D_STREAM(13, 13, 13, double, 0, 2, 352, 2, 1);
    FFT3D_STREAM_BST(13, 13, 13, double, 0, 1, 192, 3, 2);
    FFT3D_STREAM_BST(13, 13, 13, double, 0, 2, 352, 2, 1);
    FFT3D_STREAM(8, 8, 16, double, 0, 2, 128, 3, 1);
    FFT3D_STREAM(8, 8, 16, double, 0, 1, 64, 2, 4);
    // complex float
    FFT3D_STREAM(6, 6, 6, float, 0, 16, 576, 3, 1);
    FFT3D_STREAM(6, 6, 6, float, 0, 32, 1024, 2, 1);
    FFT3D_STREAM(8, 8, 8, float, 0, 8, 512, 4, 1);
    FFT3D_STREAM(8, 8, 8, float, 0, 16, 1024, 2, 1);
    FFT3D_STREAM(12, 12, 12, float, 0, 2, 288, 4, 1);
    FFT3D_STREAM(12, 12, 12, float, 0, 4, 576, 2, 1);
    FFT3D_STREAM(16, 16, 16, float, 0, 1, 256, 4, 1);
    FFT3D_STREAM_BST(16, 16, 16, float, 0, 1, 256, 4, 1);
    FFT3D_STREAM(16, 16, 16, float, 0, 2, 512, 2, 1);
    FFT3D_STREAM(17, 17, 17, float, 0, 2, 640, 2, 1);
    FFT3D_STREAM(17, 17, 17, float, 1, 2, 640, 2, 1);
    FFT3D_STREAM_BST(17, 17, 17, float, 0, 2, 640, 2, 1);
    FFT3D_STREAM_BST(17, 17, 17, float, 2, 2, 640, 2, 1);
    FFT3D_STREAM(8, 8, 16, float, 0, 4, 512, 4, 1);
    FFT3D_STREAM(8, 8, 16, float, 0, 8, 512, 2, 1);
    FFT3D_STREAM(16, 16, 32, float, 0, 1, 256, 2, 1);
    FFT3D_STREAM(16, 16, 32, float, 0, 1, 256, 3, 1);
    FFT3D_STREAM(13, 13, 13, float, 0, 2, 352, 3, 1);
    FFT3D_STREAM_BST(13, 13, 13, float, 0, 2, 352, 3, 1);
    FFT3D_STREAM(23, 23, 23, float, 0, 1, 288, 2, 1);
    FFT3D_STREAM(24, 24, 24, float, 0, 1, 576, 2, 1);
    FFT3D_STREAM(23, 23, 23, float, 0, 1, 544, 2, 1);
    FFT3D_STREAM(8, 8, 8, float, 0, 3, 192, 2, 4);
    FFT3D_STREAM(16, 16, 16, float, 0, 1, 256, 2, 1);
    FFT3D_STREAM(8, 8, 16, float, 0, 4, 128, 2, 3);
    FFT3D_STREAM(8, 8, 16, float, 0, 1, 64, 2, 8);
}

}  // namespace fft3d
