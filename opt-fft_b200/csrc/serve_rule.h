// serve_rule.h -- how the server runs the 36^3 volumes of a batch (host only;
// serve.cu, tested by hostcheck.cpp).
#pragma once

#include <algorithm>

namespace fft3d {

// Which precisions' cubes (n[0] complex double, n[1] complex float) take a list launch
// of their own (cube_list_entry) before the persistent kernel, the others being its
// items beside `other_bytes` of other volumes: of the four ways the one with the
// shortest estimate.  Measured on a B200 of 148 SMs, complex double / float: a list
// launch takes 12 us + 0.48 / 0.26 us a volume; as an item a volume holds one of the
// `sms` SMs for 98 / 49 us, beyond which the batch cannot end (items run largest
// first, and an SM takes its next item as it starts one: those with a complex double
// cube hold one of the second round's cubes too); the other kinds move 2.3 TB/s.
inline void cubes_by_list(int sms, const long long n[2], double other_bytes, bool listed[2])
{
    constexpr double launch = 12.0, list_us[2] = {0.48, 0.26}, item_us = 49.0;  // of a complex float item
    const double other = other_bytes / 2.3e6;
    double best = 0.0;
    for (int way = 0; way < 4; ++way) {
        double lists = 0.0;
        long long left[2];  // the cubes that stay in the batch
        for (int k = 0; k < 2; ++k) {
            const bool list = (way >> k & 1) != 0;
            if (list) lists += launch + list_us[k] * (double)n[k];
            left[k] = list ? 0 : n[k];
        }
        const long long last = (left[0] + sms - 1) / sms + (left[0] + left[1] + sms - 1) / sms;
        const double t = lists + std::max(item_us * (double)last,
                                          other + item_us * (double)(2 * left[0] + left[1]) / sms);
        if (way == 0 || t < best) {
            best = t;
            listed[0] = n[0] > 0 && (way & 1);
            listed[1] = n[1] > 0 && (way & 2);
        }
    }
}

}  // namespace fft3d
