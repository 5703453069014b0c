// Host part of rrtmgp_b200_kdist_create on a k-distribution with 77 scaling kinds per atmosphere, more
// than a minor-interval code holds: every interval scales with the density of another (gas,
// scaling gas) pair.  Built with the address sanitizer and run without a GPU, so creation
// ends in an allocation failure after all tables have been laid out.
#include <cstdio>
#include <string>
#include <vector>

#include "rrtmgp_b200.h"

int main()
{
    const std::vector<std::string> gas = {"h2o", "co2", "o3", "n2o", "co", "ch4", "o2", "n2", "a", "b", "c"};
    std::vector<const char*> names;
    for (const std::string& s : gas) names.push_back(s.c_str());
    const int ngas = int(names.size()), ngpt = 3, ntemp = 2, npres = 2, neta = 2, nplanck = 4;
    std::vector<const char*> minor, scaling;
    std::vector<int> lims, density, complement, start;
    for (int i = 0; i < 7; ++i)
        for (int j = 0; j < ngas; ++j) {
            const int n = int(minor.size());
            minor.push_back(names[i]);
            scaling.push_back(names[j]);
            density.push_back(1);
            complement.push_back(0);
            lims.insert(lims.end(), 2, 1 + n % ngpt);
            start.push_back(n + 1);
        }
    const int n = int(minor.size());
    const std::vector<double> kminor(size_t(ntemp) * neta * n, 1.), k(size_t(ntemp) * (npres + 1) * neta * ngpt, 1.),
        vmr(size_t(ntemp) * (ngas + 1) * 2, 1e-3), planck(nplanck, 1.);
    const int key[4] = {1, 2, 1, 2}, band[2] = {1, ngpt};
    const double press[2] = {1e5, 1e3}, temp[2] = {200., 300.};
    rrtmgp_b200_kdist_tables t{};
    t.ngas = ngas; t.nband = 1; t.ngpt = ngpt; t.ntemp = ntemp; t.npres = npres; t.neta = neta;
    t.nplanck_temp = nplanck;
    t.gas_names = names.data(); t.key_species = key; t.band_lims_gpt = band;
    t.press_ref = press; t.press_ref_trop = 1e4; t.temp_ref = temp; t.vmr_ref = vmr.data();
    t.kmajor = k.data(); t.planck_frac = k.data(); t.totplnk = planck.data();
    t.nminor_absorber = ngas; t.identifier_minor = names.data(); t.gas_minor = names.data();
    t.nint_lower = t.nint_upper = t.ncontrib_lower = t.ncontrib_upper = n;
    t.minor_gases_lower = t.minor_gases_upper = minor.data();
    t.scaling_gas_lower = t.scaling_gas_upper = scaling.data();
    t.minor_limits_gpt_lower = t.minor_limits_gpt_upper = lims.data();
    t.minor_scales_with_density_lower = t.minor_scales_with_density_upper = density.data();
    t.scale_by_complement_lower = t.scale_by_complement_upper = complement.data();
    t.kminor_start_lower = t.kminor_start_upper = start.data();
    t.kminor_lower = t.kminor_upper = kminor.data();
    rrtmgp_b200_kdist h = nullptr;
    const int st = rrtmgp_b200_kdist_create(&t, names.data(), ngas, &h);
    std::printf("status %d: %s\n", st, rrtmgp_b200_last_error());
    return st == RRTMGP_B200_ERR_ALLOC ? 0 : 1;
}
