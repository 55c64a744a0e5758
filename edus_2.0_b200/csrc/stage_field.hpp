// Field of one solve at one stage.
#pragma once

namespace edus {

// E (Cartesian, a.u.) and g = A^T E, so that R.E = g . R_crys for the
// Gamma-centred crystal coordinates R_crys.
struct StageField {
    double E[3];
    double g[3];
    double ga[3];  // Peierls gauge: A.R = ga . R_crys with A(t) the vector potential
};

}  // namespace edus
