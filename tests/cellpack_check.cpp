// Host check of csrc/cellpack.cuh: every grid that packs() accepts gives its cells back,
// at the edges of both axes and of the 16 bits; wider grids are refused.
#include <cstdio>
#include <initializer_list>

#include "../mps_gb300/csrc/cellpack.cuh"

using namespace mpsg;

int main() {
    const int dims[] = {1, 2, 28, 32767, 32768, 32769, 33901, 65535, 65536, 65537, 110000, 1 << 30};
    int bad = 0, refused = 0;
    for (int nx : dims)
        for (int ny : dims) {
            if (packs(nx, ny) != (nx <= 1 << 16 && ny <= 1 << 16)) bad++;
            if (!packs(nx, ny)) {
                refused++;
                continue;
            }
            for (int x : {0, 1, nx / 2, nx - 2, nx - 1})
                for (int y : {0, 1, ny / 2, ny - 2, ny - 1}) {
                    if (x < 0 || y < 0 || x >= nx || y >= ny) continue;
                    const uint32_t c = pack_cell(x, y);
                    if (cell_x(c) != x || cell_y(c) != y) bad++;
                }
        }
    std::printf("%d wrong, %d refused\n", bad, refused);
    return bad || refused != 12 * 12 - 9 * 9;
}
