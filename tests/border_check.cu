// The index checks of the pair sweep's slow path (border_in), on the host: the
// position arrays count every read outside [0, n).
#include <cstdio>

#include "dm_pair.cuh"

static int g_outside = 0;

struct Checked {
    const double *v;
    int n;
    double operator[](int i) const {
        if (i < 0 || i >= n) {
            g_outside++;
            return 0.0;
        }
        return v[i];
    }
};

struct HostView {
    Checked x, y;
    Checked px() const { return x; }
    Checked py() const { return y; }
    double kappa() const { return 2e4; }  // cutoff 5e-4
};

int main() {
    const double x[3] = {0.0, 4.9e-4, 5.1e-4}, y[3] = {0.0, 0.0, 0.0};
    const HostView P{{x, 3}, {y, 3}};
    const bool want[4][4] = {{false, false, false, false},   // i = -1
                             {false, false, true, false},    // i = 0 (columns: j = -1, 0, 1, 2)
                             {false, true, false, true},
                             {false, false, true, false}};
    int wrong = 0;
    for (int i = -1; i < 3; i++)
        for (int j = -1; j < 3; j++) wrong += dm::border_in(P, i, j) != want[i + 1][j + 1];
    std::printf("wrong %d outside %d\n", wrong, g_outside);
    return wrong || g_outside;
}
