// Host-side check of the rule that chooses between the two prefill attention kernels (attention_tc_faster, csrc/common.cuh): its lines lie at the
// same occupancy whatever the number of SMs.  Runs on the CPU; no GPU code is launched.
#include <cstdio>

#include "common.cuh"

using sbvr::attention_tc_faster;

int main() {
    int failures = 0;
    auto check = [&](bool got, bool want, const char* what, int sms) {
        if (got != want) ++failures, std::printf("%s at %d SMs\n", what, sms);
    };
    check(attention_tc_faster(96, 128, 148), true, "96 blocks of a prompt of 128", 148);
    check(attention_tc_faster(95, 128, 148), false, "95 blocks of a prompt of 128", 148);
    for (int sms : {20, 74, 132, 148, 160}) {
        check(attention_tc_faster(1, 256, sms), true, "a prompt of 256", sms);
        check(attention_tc_faster(2 * sms, 64, sms), false, "two blocks per SM", sms);
        check(attention_tc_faster(2 * sms + 1, 64, sms), true, "a block more than two per SM", sms);
        check(attention_tc_faster(sms, 128, sms), true, "a block per SM", sms);
        check(attention_tc_faster(sms / 2, 128, sms), false, "a block per two SMs", sms);
    }
    std::printf("%d failures\n", failures);
    return failures != 0;
}
