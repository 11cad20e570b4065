// hostcheck.cu -- a host build of the pointwise right-hand side (physics.cuh) and of its
// hand-written adjoint (adjoint.cuh), so the adjoint can be checked against finite
// differences of the forward map without a GPU.  Built into libsunset_hostcheck.so; the time
// step itself never calls it.
#include <algorithm>
#include <utility>
#include <vector>

#include "adjoint.cuh"
#include "device_blocks.h"

extern "C" {

// par: Re, Wi, beta, epsPTT, Ma.  s[6], g[18] as in adjoint.cuh; r[6] = P(s, g); with rbar
// given, sbar[6], gbar[18], tbar[2] (Wi, beta) = rbar^T dP.
int sunset_hostcheck_lc(const double *par, const double *s, const double *g, int first, const double *rbar,
                        double *r, double *sbar, double *gbar, double *tbar) {
    SunsetConfig c{};
    c.form = SUNSET_FORM_LC;
    c.morder = c.forder = 6;
    c.kolmogorov_forcing = 0;
    c.L_char = 1.0;
    c.U_char = 1.0;
    c.Re = par[0];
    c.Wi = par[1];
    c.beta = par[2];
    c.epsPTT = par[3];
    c.Ma = par[4];
    c.fenep_l2 = 1e30;
    const sunset::StepConsts K = sunset::step_consts(c, 1, 1, false, false);
    sunset::p_forward_lc(K, s, g, first != 0, 0.0, r);
    if (rbar) {
        for (int k = 0; k < sunset::kAdjS; k++) sbar[k] = 0.0;
        for (int k = 0; k < sunset::kAdjG; k++) gbar[k] = 0.0;
        tbar[0] = tbar[1] = 0.0;
        sunset::p_adjoint_lc(K, s, g, first != 0, rbar, sbar, gbar, tbar);
    }
    return 0;
}

// deal_slice_by_bank (bank_deal.cu) on one slice given as flat lists: lane r's small entries
// are small[soff[r] .. soff[r + 1]), its other entries large[loff[r] .. loff[r + 1]); pos[e] is
// the local position of entry e.  chosen[k * 32 + lane] for k < width (-1: padding).
int sunset_hostcheck_deal(int group, const uint16_t *pos, const int *small, const int *soff, const int *large,
                          const int *loff, int width, int *chosen) {
    std::vector<int> vs[sunset::kSlice], vl[sunset::kSlice];
    int c_s[sunset::kSlice], c[sunset::kSlice];
    for (int r = 0; r < sunset::kSlice; r++) {
        vs[r].assign(small + soff[r], small + soff[r + 1]);
        vl[r].assign(large + loff[r], large + loff[r + 1]);
        c_s[r] = (int)vs[r].size();
        c[r] = c_s[r] + (int)vl[r].size();
    }
    sunset::deal_slice_by_bank(group, pos, vs, vl, c_s, c, width, chosen);
    return 0;
}

// The handle's memory blocks (device_blocks.h) over a pretended device of `limit` bytes, whose
// addresses are only numbers.  Operation k: size[k] > 0 takes that many bytes, address[k] gets the
// piece's address (0: refused); size[k] <= 0 gives back the piece of operation -size[k].  held[k]:
// bytes the blocks take from the device after it; calls[k]: how often the device was asked so far.
// Returns the bytes still taken after everything is cleared, or the last refusal's error code if
// that is 0 (42: out of memory).
namespace {
struct FakeDevice {
    size_t limit, held, next;
    int calls;
    std::vector<std::pair<char *, size_t>> given;
} fake;
int fake_acquire(void **p, size_t bytes) {
    fake.calls++;
    if (fake.held + bytes > fake.limit) return 42;
    *p = reinterpret_cast<char *>(fake.next);
    fake.given.push_back({static_cast<char *>(*p), bytes});
    fake.next += bytes + 4096;
    fake.held += bytes;
    return 0;
}
void fake_release(void *p) {
    for (auto &g : fake.given)
        if (g.first == p) {
            fake.held -= g.second;
            g.first = nullptr;
            return;
        }
    fake.held = (size_t)1 << 62;  // given back twice, or never taken
}
}  // namespace
int sunset_hostcheck_blocks(long long limit, int n, const long long *size, long long *address, long long *held, int *calls) {
    fake = {(size_t)limit, 0, (size_t)1 << 40, 0, {}};
    sunset::DeviceBlocks B;
    B.acquire = fake_acquire;
    B.release = fake_release;
    for (int k = 0; k < n; k++) {
        if (size[k] > 0) address[k] = (long long)reinterpret_cast<size_t>(B.take((size_t)size[k]));
        else B.give(reinterpret_cast<char *>((size_t)address[-size[k]]));
        held[k] = (long long)fake.held;
        calls[k] = fake.calls;
    }
    B.clear();
    return fake.held ? (int)std::min(fake.held, (size_t)1 << 30) : B.error;
}

// c = lc_c_from_psi(psi) and, with cbar given, psibar = cbar^T dc/dpsi.
int sunset_hostcheck_lc_c(const double *psi, const double *cbar, double *c, double *psibar) {
    sunset::lc_c_from_psi(psi[0], psi[1], psi[2], &c[0], &c[1], &c[2]);
    if (cbar) {
        psibar[0] = psibar[1] = psibar[2] = 0.0;
        sunset::lc_c_from_psi_adj(psi[0], psi[1], psi[2], cbar, psibar);
    }
    return 0;
}
}
