// Host check of film_tiles (device_types.h).

#include "../raycer_gb300/csrc/device_types.h"

#include <cstdio>

namespace
{

int failures = 0;
#define CHECK(x)                                        \
    do                                                  \
    {                                                   \
        if (!(x))                                       \
        {                                               \
            std::printf("line %d: %s\n", __LINE__, #x); \
            failures++;                                 \
        }                                               \
    } while (0)

// The largest films are taken in tiles too, as long as a queue head's 32 bits
// hold the tiles' pixels and what 2^19 warps take past them.
void largest_films()
{
    const int64_t pixels[] = { (int64_t(1) << 30) - 1024, int64_t(1) << 30, (int64_t(1) << 30) + 1024, int64_t(1) << 31 };
    const int64_t widths[] = { 32768, 1024, 9, 8 };
    for (int64_t width : widths)
        for (int64_t n : pixels)
        {
            const int64_t count = n / width * width;
            const rcx::FilmTiles t = rcx::film_tiles(0, count, width);
            const int64_t columns = (width + 7) / 8, rows = (count / width + 3) / 4;
            if (32 * columns * rows < (int64_t(1) << 32) - (int64_t(1) << 24))
                CHECK(t.columns == columns && t.rows == rows && t.width == width && t.skip == 0);
            else
                CHECK(t.columns == 0);
        }
    CHECK(rcx::film_tiles(0, int64_t(1) << 31, 32768).columns == 4096);
    CHECK(rcx::film_tiles(0, (int64_t(1) << 30) * 2 - 2, 9).columns == 2);
}

}  // namespace

int main()
{
    largest_films();
    if (!failures)
        std::printf("film tiles ok\n");
    return failures ? 1 : 0;
}
