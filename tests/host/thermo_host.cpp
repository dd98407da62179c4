// Host build of the moments' temperature iteration (csrc/gas.cuh), for tests/test_temperature_iteration.py.
#include "gas.cuh"

namespace {
template <int NS>
int solve(const lbmgpu_mech *m, int fast, const double *Y, double u, double T0, double *T) {
    gas::Tables t{};
    gas::make_tables_base(*m, t);
    gas::ThermoTab<NS> tab;
    tab.fill(t, 0, 1);
    return fast ? gas::T_from_u_tab<NS, true>(tab, Y, u, T0, *T) : gas::T_from_u_tab<NS, false>(tab, Y, u, T0, *T);
}
}  // namespace

extern "C" {
double energy(const lbmgpu_mech *m, const double *Y, double T) {
    gas::Tables t{};
    gas::make_tables_base(*m, t);
    return gas::int_energy_mass(t, Y, T);
}
int temperature(const lbmgpu_mech *m, int fast, const double *Y, double u, double T0, double *T) {
    return m->n_species == 9 ? solve<9>(m, fast, Y, u, T0, T) : solve<6>(m, fast, Y, u, T0, T);
}
}
