// stream_odd_kernels.cu -- the STREAM kernels (stream.cuh) of the other extents:
// small and odd cubes and anisotropic volumes.
//
// The VOLUME kernels of these extents load a group of volumes, transform it and
// store it with one CTA resident, or a few, so HBM idles while they compute and
// the reverse: 25-60% of the copy rate.  Here the next item's load is in flight
// during an item's passes, items are 8-50 KB so that 2-8 CTAs share an SM, and
// odd n2 (natural layout) moves whole items by bulk copies both ways.  Measured
// on B200 over 96 MB (floor 30 us at 6.65 TB/s; a device copy takes 34.4 us),
// VOLUME against STREAM: 9x25x7 c128 115 / 36.8 us, 11x4x9 81.9 / 35.9, 25x4x3
// 82.4 / 37.0, 7x11x13 63.8 / 36.0, 15^3 59.9 / 37.7, 24x18x12 73.8 / 50.5,
// 1x1x16 c64 125 / 33.8, 9x25x7 c64 95.4 / 37.0, 7x11x13 c64 68.5 / 38.1, 1^3 102 /
// 33.5, 8x8x1 (as 1x8x8) c128 66.9 / 35.7 and c64 48.4 / 39.0.  Of some
// 900 shapes swept (2-4 stages, 1-8 CTAs an SM, register or bulk stores) the
// fastest of each extent is kept, and a second one with smaller items where that
// costs under 7%, for batches that the larger items would leave on few SMs.  (4^3
// complex double and 8x1x8 complex float have VOLUME alone.)  The
// VOLUME kernels stay in the tuner's race: at under a few hundred volumes their
// one pass per CTA is up to 20% shorter (9x25x7 c128 x 20: 3.5 / 4.1 us).
#include "stream.cuh"

namespace fft3d {

void register_stream_odd_kernels(std::vector<KernelEntry> &out)
{
    // complex double
    FFT3D_STREAM_BST(1, 1, 1, double, 0, 1024, 256, 2, 4);
    FFT3D_STREAM(2, 2, 2, double, 0, 72, 160, 2, 8);
    FFT3D_STREAM(3, 3, 3, double, 0, 21, 192, 3, 4);
    FFT3D_STREAM_BST(5, 5, 5, double, 0, 9, 128, 3, 2);
    FFT3D_STREAM_BST(7, 7, 7, double, 0, 3, 160, 3, 2);
    FFT3D_STREAM_BST(9, 9, 9, double, 0, 1, 96, 4, 4);
    FFT3D_STREAM(10, 10, 10, double, 0, 1, 128, 2, 2);
    FFT3D_STREAM_BST(11, 11, 11, double, 0, 1, 128, 3, 1);
    FFT3D_STREAM_BST(15, 15, 15, double, 0, 1, 256, 2, 1);
    FFT3D_STREAM_BST(2, 3, 5, double, 0, 59, 192, 2, 4);
    FFT3D_STREAM_BST(2, 3, 5, double, 0, 28, 96, 2, 8);
    FFT3D_STREAM_BST(7, 11, 13, double, 0, 1, 96, 2, 4);
    FFT3D_STREAM(5, 8, 12, double, 0, 2, 96, 2, 3);
    FFT3D_STREAM(5, 8, 12, double, 0, 1, 64, 2, 8);
    FFT3D_STREAM(13, 5, 8, double, 0, 2, 96, 3, 4);
    FFT3D_STREAM_BST(13, 5, 8, double, 0, 1, 64, 2, 4);
    FFT3D_STREAM(17, 2, 2, double, 0, 17, 96, 2, 2);
    FFT3D_STREAM(32, 8, 4, double, 0, 1, 64, 2, 3);
    FFT3D_STREAM(1, 8, 8, double, 0, 13, 128, 2, 4);
    FFT3D_STREAM_BST(8, 1, 8, double, 0, 13, 128, 4, 4);
    FFT3D_STREAM_FLAT(8, 8, double, 13, 128, 2, 4);
    FFT3D_STREAM_BST(49, 2, 2, double, 0, 8, 64, 2, 3);
    FFT3D_STREAM_BST(25, 4, 3, double, 0, 5, 64, 2, 4);
    FFT3D_STREAM(27, 2, 2, double, 0, 7, 64, 3, 2);
    FFT3D_STREAM(19, 3, 2, double, 0, 5, 64, 2, 4);
    FFT3D_STREAM_BST(23, 2, 2, double, 0, 12, 64, 2, 4);
    FFT3D_STREAM(1, 1, 16, double, 0, 54, 64, 2, 8);
    FFT3D_STREAM_BST(1, 7, 1, double, 0, 170, 192, 3, 2);
    FFT3D_STREAM_BST(3, 5, 7, double, 0, 11, 96, 2, 3);
    FFT3D_STREAM_BST(3, 5, 7, double, 0, 5, 96, 3, 4);
    FFT3D_STREAM(4, 6, 10, double, 0, 3, 96, 2, 4);
    FFT3D_STREAM_BST(16, 3, 5, double, 0, 3, 64, 2, 8);
    FFT3D_STREAM(24, 18, 12, double, 0, 1, 224, 2, 1);
    FFT3D_STREAM(2, 2, 64, double, 0, 14, 64, 2, 2);
    FFT3D_STREAM_BST(64, 2, 2, double, 0, 6, 64, 2, 3);
    FFT3D_STREAM_BST(9, 25, 7, double, 0, 1, 64, 2, 4);
    FFT3D_STREAM(20, 12, 6, double, 0, 1, 96, 2, 2);
    FFT3D_STREAM_BST(11, 4, 9, double, 0, 2, 64, 2, 4);
    // complex float
    FFT3D_STREAM_BST(1, 1, 1, float, 0, 2048, 256, 2, 4);
    FFT3D_STREAM(2, 2, 2, float, 0, 148, 320, 2, 4);
    FFT3D_STREAM_BST(3, 3, 3, float, 0, 88, 512, 3, 2);
    FFT3D_STREAM(4, 4, 4, float, 0, 44, 512, 2, 2);
    FFT3D_STREAM(4, 4, 4, float, 0, 22, 192, 2, 4);
    FFT3D_STREAM_BST(5, 5, 5, float, 0, 28, 352, 2, 4);
    FFT3D_STREAM_BST(7, 7, 7, float, 0, 10, 256, 2, 2);
    FFT3D_STREAM_BST(9, 9, 9, float, 0, 2, 96, 2, 4);
    FFT3D_STREAM(10, 10, 10, float, 0, 2, 224, 2, 3);
    FFT3D_STREAM_BST(10, 10, 10, float, 0, 1, 128, 2, 8);
    FFT3D_STREAM_BST(11, 11, 11, float, 0, 2, 128, 2, 4);
    FFT3D_STREAM_BST(15, 15, 15, float, 0, 2, 256, 2, 2);
    FFT3D_STREAM_BST(2, 3, 5, float, 0, 59, 192, 2, 4);
    FFT3D_STREAM(7, 11, 13, float, 0, 2, 96, 2, 3);
    FFT3D_STREAM(5, 8, 12, float, 0, 3, 128, 2, 4);
    FFT3D_STREAM(13, 5, 8, float, 0, 4, 160, 2, 3);
    FFT3D_STREAM(13, 5, 8, float, 0, 2, 96, 2, 8);
    FFT3D_STREAM(17, 2, 2, float, 0, 17, 96, 2, 8);
    FFT3D_STREAM_BST(32, 8, 4, float, 0, 1, 64, 3, 2);
    FFT3D_STREAM(1, 8, 8, float, 0, 33, 160, 2, 3);
    FFT3D_STREAM_FLAT(8, 8, float, 33, 160, 2, 3);
    FFT3D_STREAM(49, 2, 2, float, 0, 6, 64, 2, 4);
    FFT3D_STREAM_BST(25, 4, 3, float, 0, 5, 64, 2, 8);
    FFT3D_STREAM_BST(27, 2, 2, float, 0, 10, 64, 2, 8);
    FFT3D_STREAM(19, 3, 2, float, 0, 21, 128, 2, 2);
    FFT3D_STREAM(19, 3, 2, float, 0, 10, 64, 2, 4);
    FFT3D_STREAM_BST(23, 2, 2, float, 0, 26, 128, 2, 2);
    FFT3D_STREAM_BST(23, 2, 2, float, 0, 12, 64, 2, 8);
    FFT3D_STREAM(1, 1, 16, float, 0, 224, 224, 2, 2);
    FFT3D_STREAM_BST(1, 7, 1, float, 0, 256, 128, 2, 4);
    FFT3D_STREAM_BST(3, 5, 7, float, 0, 22, 192, 3, 2);
    FFT3D_STREAM(4, 6, 10, float, 0, 9, 128, 2, 3);
    FFT3D_STREAM_BST(16, 3, 5, float, 0, 9, 160, 2, 3);
    FFT3D_STREAM(24, 18, 12, float, 0, 1, 224, 2, 2);
    FFT3D_STREAM(2, 2, 64, float, 0, 14, 64, 2, 2);
    FFT3D_STREAM(2, 2, 64, float, 0, 6, 64, 2, 4);
    FFT3D_STREAM(64, 2, 2, float, 0, 4, 64, 2, 4);
    FFT3D_STREAM_BST(9, 25, 7, float, 0, 2, 128, 2, 2);
    FFT3D_STREAM_BST(20, 12, 6, float, 0, 1, 96, 2, 4);
    FFT3D_STREAM(11, 4, 9, float, 0, 4, 160, 2, 4);
}

}  // namespace fft3d
