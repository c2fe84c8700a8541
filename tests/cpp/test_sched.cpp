// Host unit test of the pass schedules a context keeps per image size
// (glscv_gb300/csrc/sched_internal.h), compiled without nvcc.
#include <cstdio>
#include <map>

#include "sched_internal.h"

using namespace glsfft;

static int failures = 0;
#define CHECK(c)                                                   \
    do {                                                           \
        if (!(c)) {                                                \
            std::printf("FAIL line %d: %s\n", __LINE__, #c);        \
            failures++;                                            \
        }                                                          \
    } while (0)

int main() {
    // 2048-point rows: the small-grid schedule up to 1024 rows of a launch,
    // however they divide into images
    CHECK(default_schedule(1024, 2048).row == 3 && default_schedule(2048, 2048).row == 2);
    for (int rows = 1; rows <= 4096; rows *= 2)
        for (int images : {1, 2, 3, 7, 8, 16, 50, 65535})
            CHECK(default_schedule(rows, 2048, images).row == ((long long)rows * images <= 1024 ? 3 : 2));
    // other lengths do not depend on the number of images
    for (int cols = 1; cols <= 4096; cols *= 2)
        for (int images : {1, 50})
            if (cols != 2048) CHECK(default_schedule(512, cols, images).row == (cols == 4096 ? 2 : 0));

    std::map<long long, FftSchedule> m;
    CHECK(schedule_for(m, 512, 2048).row == 3 && schedule_for(m, 512, 2048, 50).row == 2);
    // setting the built-in pair brings the built-in choice back
    keep_schedule(m, 512, 2048, FftSchedule{1, 0});
    CHECK(schedule_for(m, 512, 2048, 50).row == 1);
    keep_schedule(m, 512, 2048, FftSchedule{3, 0});
    CHECK(m.empty());
    // a pair tuned on many images is what runs and what is reported
    for (int row : {2, 3}) {
        keep_schedule(m, 512, 2048, FftSchedule{row, 0}, 50);
        CHECK(schedule_for(m, 512, 2048).row == row && schedule_for(m, 512, 2048, 50).row == row);
    }
    // one launch for both passes: a pair of passes must beat it by the margin
    // and be one that runs when it is set
    const FftSchedule d = default_schedule(64, 64), other{1, 0};
    CHECK(one_launch_stays(1.0, 1.5, other, d, 0.01) && one_launch_stays(1.0, 0.995, other, d, 0.01));
    CHECK(!one_launch_stays(1.0, 0.9, other, d, 0.01));
    CHECK(one_launch_stays(1.0, 0.9, d, d, 0.01));

    std::printf(failures ? "%d FAILED\n" : "ALL OK\n", failures);
    return failures != 0;
}
