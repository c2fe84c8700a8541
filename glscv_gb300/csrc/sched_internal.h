// sched_internal.h -- the selectable schedules of the plain path's complex
// row and column passes, and the per-size choice a context keeps.
#pragma once
#include <cuda_runtime.h>

#include "fft_config.h"
#include "glsfft_internal.h"

namespace glsfft {

// id 0..kPassSchedules-1 of fft_config.h; unavailable ids give
// cudaErrorInvalidValue without launching
cudaError_t launch_rows_sched(int n, int id, const PassArgs &a, int images, cudaStream_t s);
cudaError_t launch_cols_sched(int n, int id, const PassArgs &a, int images, cudaStream_t s);

struct FftSchedule {
    int row = 0;  // schedule of the row pass (line length cols)
    int col = 0;  // schedule of the column pass (line length rows)
};
inline long long sched_key(int rows, int cols) { return ((long long)rows << 20) | cols; }

// The schedules `images` images of a size run in one launch until the size is
// set or tuned otherwise, from measurements on GB300: schedule 2 for 2048- and
// 4096-point rows (one 4096^2 image, per pass: 45 us, as schedule 0, and ahead
// of it on fewer rows), schedule 3 for up to 1024 2048-point rows in all (row
// pass, schedule 2 / 3: 64 rows 3.1 / 2.5 us, 512 4.6 / 4.5, 1024 6.9 / 6.5,
// 2048 10.5 / 10.7, 4096 23.0 / 24.3, 25600 120 / 130), and the streamed pass
// for 4096-point columns (68 us against 91); other lengths run schedule 0.
inline FftSchedule default_schedule(int rows, int cols, int images = 1) {
    FftSchedule s{};
    if (cols == 2048 || cols == 4096) s.row = 2;
    if (cols == 2048 && (long long)rows * images <= 1024) s.row = 3;
    if (rows == 4096) s.col = kSchedStreamed;
    return s;
}
template <class Map>
inline FftSchedule schedule_for(const Map &m, int rows, int cols, int images = 1) {
    const auto it = m.find(sched_key(rows, cols));
    return it != m.end() ? it->second : default_schedule(rows, cols, images);
}
// Sizes that run both passes in one launch by default: whether that stays when
// the tuner's best pair of passes `two` took two_ms and the one launch one_ms.
// It does unless the pair is faster by `margin`, and when the pair is the
// default one, which cannot be asked for apart from it.
inline bool one_launch_stays(double one_ms, double two_ms, FftSchedule two, FftSchedule dflt,
                             double margin) {
    return two_ms >= one_ms * (1.0 - margin) || (two.row == dflt.row && two.col == dflt.col);
}
// Keep `s`, chosen for `images` images, for a size: the built-in choice needs
// no entry, but a choice that differs for one image is kept as made.
template <class Map>
inline void keep_schedule(Map &m, int rows, int cols, FftSchedule s, int images = 1) {
    auto same = [&](const FftSchedule &d) { return s.row == d.row && s.col == d.col; };
    if (same(default_schedule(rows, cols)) && same(default_schedule(rows, cols, images)))
        m.erase(sched_key(rows, cols));
    else
        m[sched_key(rows, cols)] = s;
}

}  // namespace glsfft
