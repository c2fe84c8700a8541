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

// The schedules an image size runs until it is set or tuned otherwise,
// from measurements on GB300: schedule 2 for 2048- and 4096-point rows (one
// 4096^2 image, per pass: 45 us, as schedule 0, and ahead of it on fewer rows),
// schedule 3 for up to 1024 2048-point rows (1024 x 2048 forward + inverse
// 27.5 us against 29.3), and the streamed pass for 4096-point columns (68 us
// against 91); other lengths run schedule 0.
inline FftSchedule default_schedule(int rows, int cols) {
    FftSchedule s{};
    if (cols == 2048 || cols == 4096) s.row = 2;
    if (cols == 2048 && rows <= 1024) s.row = 3;
    if (rows == 4096) s.col = kSchedStreamed;
    return s;
}
template <class Map>
inline FftSchedule schedule_for(const Map &m, int rows, int cols) {
    const auto it = m.find(sched_key(rows, cols));
    return it != m.end() ? it->second : default_schedule(rows, cols);
}

}  // namespace glsfft
