// Host check of film_tiles and tile_pixels_before (device_types.h).

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

// tile_pixels_before against the tiles' pixels counted one by one.
void pixels_before()
{
    const int64_t widths[] = { 8, 9, 15, 16, 37 };
    const int64_t starts[] = { 0, 1, 8, 30 };
    const int64_t counts[] = { 37 * 4, 301, 555 };
    for (int64_t width : widths)
        for (int64_t start : starts)
            for (int64_t count : counts)
            {
                const rcx::FilmTiles t = rcx::film_tiles(uint64_t(start), count, width);
                CHECK(t.columns > 0);
                int64_t n = 0;
                for (int64_t tile = 0; tile < int64_t(t.columns) * t.rows; ++tile)
                {
                    CHECK(rcx::tile_pixels_before(t, count, tile) == n);
                    for (int64_t k = 0; k < 32; ++k)
                    {
                        const int64_t x = tile % t.columns * 8 + k % 8, y = tile / t.columns * 4 + k / 8;
                        const int64_t i = y * width + x - t.skip;
                        n += x < width && i >= 0 && i < count ? 1 : 0;
                    }
                }
                CHECK(n == count);
                CHECK(rcx::tile_pixels_before(t, count, int64_t(t.columns) * t.rows) == count);
            }
}

}  // namespace

int main()
{
    largest_films();
    pixels_before();
    if (!failures)
        std::printf("film tiles ok\n");
    return failures ? 1 : 0;
}
