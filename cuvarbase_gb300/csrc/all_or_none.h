// Host objects that are made together or not at all.
#pragma once

namespace cuvgls {

// Makes a[0 .. n) with make(&a[i]); when one fails (make returns false), drops
// those made before it, sets all to null and returns false.
template <typename T, typename Make, typename Drop>
bool make_all(T *a, int n, Make make, Drop drop) {
    for (int i = 0; i < n; ++i) {
        if (make(&a[i])) continue;
        while (i-- > 0) drop(a[i]);
        for (int k = 0; k < n; ++k) a[k] = T{};
        return false;
    }
    return true;
}

}  // namespace cuvgls
