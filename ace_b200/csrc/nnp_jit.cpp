// nnp_jit.cpp -- symmetry-function and force kernels specialised at run time
// for the loaded potential.
//
// The prebuilt kernels read every angular function's (lambda, zeta, eta) from
// memory and branch on them per pair.  Here the host writes CUDA source in
// which each angular block of the potential is straight-line code: the
// bases 0.5 +- 0.5 cos, their powers as a shared multiply ladder, the radial
// factors once per width, and every parameter a literal.  NVRTC compiles it
// for sm_100a when the handle is created; the kernels reuse the per-atom
// skeleton of nnp_device.cuh (symm_body / force_body) through a Blocks policy,
// so only the block arithmetic differs from the prebuilt path.
#include <cuda_runtime.h>
#include <nvrtc.h>

#include <sys/stat.h>
#include <unistd.h>

#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <fstream>
#include <iterator>
#include <map>
#include <mutex>
#include <set>
#include <sstream>
#include <string>
#include <system_error>
#include <thread>
#include <vector>

#include "nnp_engine.h"

namespace nnp {

extern const char *const kDeviceHeaderSource;    // nnp_device.cuh, embedded at build time
extern const char *const kMomentsHeaderSource;   // nnp_moments.cuh

namespace {

std::string flit(float x)
{
    char b[64];
    std::snprintf(b, sizeof b, "%.9ef", x);
    return b;
}

struct Fn {
    float lf, zeta, ieta2;
    int damp, iz;
};

// emits x_b^n (n >= 1 integer) from a binary ladder, memoised
struct Powers {
    std::ostringstream &os;
    std::set<std::string> done;
    explicit Powers(std::ostringstream &o) : os(o) {}
    std::string ladder(int b, int e)   // x_b^(2^e)
    {
        const std::string name = "x" + std::to_string(b) + "_" + std::to_string(1 << e);
        if (e == 0) return "x" + std::to_string(b);
        if (!done.count(name)) {
            const std::string h = ladder(b, e - 1);
            os << "            const float " << name << " = " << h << " * " << h << ";\n";
            done.insert(name);
        }
        return name;
    }
    std::string pw(int b, int n)
    {
        if (n == 0) return "1.0f";
        std::vector<std::string> terms;
        for (int e = 0; (1 << e) <= n; ++e)
            if (n & (1 << e)) terms.push_back(ladder(b, e));
        if (terms.size() == 1) return terms[0];
        const std::string name = "x" + std::to_string(b) + "p" + std::to_string(n);
        if (!done.count(name)) {
            os << "            const float " << name << " = " << terms[0];
            for (size_t k = 1; k < terms.size(); ++k) os << " * " << terms[k];
            os << ";\n";
            done.insert(name);
        }
        return name;
    }
    // x_b^zeta for any zeta: ladder when integer, exp2/log2 otherwise
    std::string power(int b, float zeta, int iz)
    {
        if (iz >= 0) return pw(b, iz);
        const std::string name = "x" + std::to_string(b) + "r" + std::to_string(done.size());
        os << "            const float " << name << " = (x" << b << " > 0.f) ? exp2f(" << flit(zeta) << " * log2f(x" << b
           << ")) : 0.f;\n";
        done.insert(name);
        return name;
    }
};

std::vector<Fn> block_fns(const Engine &E, const DevBlockA &B)
{
    std::vector<Fn> fs;
    for (int f = 0; f < B.n; ++f) {
        const float4 q = E.apar_host[B.par + f];
        int pk;
        std::memcpy(&pk, &q.w, sizeof pk);
        fs.push_back({q.x, q.y, q.z, pk & 0xff, (pk >> 8) - 1});
    }
    // radial groups: GAUSS has its damping factors, the other forms one per width
    if (B.form != ANG_GAUSS) {
        std::vector<float> widths;
        for (Fn &f : fs) {
            size_t g = 0;
            while (g < widths.size() && widths[g] != f.ieta2) ++g;
            if (g == widths.size()) widths.push_back(f.ieta2);
            f.damp = (int)g;
        }
    }
    return fs;
}

// bases x_b = |1/2 + lambda/2 cos| of a block's functions
void gen_bases(std::ostringstream &os, const std::vector<Fn> &fs, std::vector<float> &bases)
{
    for (const Fn &f : fs) {
        bool seen = false;
        for (float x : bases) seen |= (x == f.lf);
        if (!seen) bases.push_back(f.lf);
    }
    for (size_t b = 0; b < bases.size(); ++b)
        os << "            const float x" << b << " = fabsf(fmaf(" << flit(bases[b]) << ", cs, 0.5f));\n";
}

// Common per-pair prologue: geometry, bases, and for each radial group g of
// the block its value P_g (for GAUSS the product of the two neighbours' staged
// damping factors, for the other forms the radial factor times both cutoffs,
// angular_generic's formulas with the width as a literal, once for all
// functions that share it) and, with der, its derivatives A_g, B_g with respect
// to the two distances.
void pair_prologue(std::ostringstream &os, const DevBlockA &B, const std::vector<Fn> &fs, std::vector<float> &bases,
                   std::set<int> &groups, bool der)
{
    os << "            int a, b;\n"
          "            pit_slots(k, it, a, b);\n"
          "            const float4 ua = v.u[a], ub = v.u[b];\n"
          "            const float cs = ua.x * ub.x + ua.y * ub.y + ua.z * ub.z;\n";
    gen_bases(os, fs, bases);
    for (const Fn &f : fs) groups.insert(f.damp);
    if (B.form != ANG_GAUSS) {
        const std::string c = std::to_string(B.cut);
        os << "            const float ra = v.r[a], rb = v.r[b], ca = v.fc[" << c << " * cap + a], cb = v.fc[" << c
           << " * cap + b], r2 = fmaf(ra, ra, rb * rb), cc = ca * cb;\n";
        if (der)
            os << "            const float ga = v.fd[" << c << " * cap + a], gb = v.fd[" << c << " * cap + b];\n";
        for (int g : groups) {
            float w = 0.f;
            for (const Fn &f : fs)
                if (f.damp == g) w = f.ieta2;
            const std::string G = std::to_string(g);
            const float pw = 0.5f * 3.14159265358979f * w;
            std::string df;                                       // d(rad)/dr = -2 r df rad
            if (B.form == ANG_GAUSS2 || B.form == ANG_SECH) {
                const bool sech = B.form == ANG_SECH;
                os << "            const float f" << G << " = expf(" << flit(-pw) << " * r2), n" << G << " = 1.f / (1.f + f" << G
                   << (sech ? " * f" + G : std::string()) << "), h" << G << " = 2.f * f" << G << " * n" << G << ";\n";
                df = flit(pw) + " * n" + G + (sech ? " * (1.f - f" + G + " * f" + G + ")" : "");
            } else {
                const int e = 4 + (B.form - ANG_STUDENT3);
                os << "            const float n" << G << " = rsqrtf(fmaf(" << flit(w) << ", r2, 1.f)), h" << G << " = ipow(n" << G
                   << ", " << e << ");\n";
                df = flit(0.5f * (float)e * w) + " * n" + G + " * n" + G;
            }
            os << "            const float P" << G << " = h" << G << " * cc;\n";
            if (der)
                os << "            const float d" << G << " = -2.f * " << df << ", A" << G << " = h" << G << " * cb * fmaf(ra * ca, d"
                   << G << ", ga), B" << G << " = h" << G << " * ca * fmaf(rb * cb, d" << G << ", gb);\n";
        }
        return;
    }
    // damping factors: groups 2m and 2m+1 of a neighbour are one float2 (wix)
    std::set<int> pairs;
    for (int d : groups) pairs.insert(d >> 1);
    for (int m : pairs) {
        const std::string M = std::to_string(m);
        os << "            const float2 wpa" << M << " = reinterpret_cast<const float2 *>(v.w)[" << M
           << " * cap + a], wpb" << M << " = reinterpret_cast<const float2 *>(v.w)[" << M << " * cap + b];\n";
        if (der)
            os << "            const float2 dpa" << M << " = reinterpret_cast<const float2 *>(v.wd)[" << M
               << " * cap + a], dpb" << M << " = reinterpret_cast<const float2 *>(v.wd)[" << M << " * cap + b];\n";
    }
    for (int d : groups) {
        const std::string M = std::to_string(d >> 1), c = (d & 1) ? ".y" : ".x", D = std::to_string(d);
        os << "            const float P" << D << " = wpa" << M << c << " * wpb" << M << c << ";\n";
        if (der)
            os << "            const float A" << D << " = dpa" << M << c << " * wpb" << M << c << ", B" << D << " = wpa" << M << c
               << " * dpb" << M << c << ";\n";
    }
}

int base_of(const std::vector<float> &bases, float lf)
{
    for (size_t b = 0; b < bases.size(); ++b)
        if (bases[b] == lf) return (int)b;
    return 0;
}

// Sums over the warp of the per-lane accumulators s0 .. s(nf-1), stored to
// dst[f] by one lane each.  The list (padded with zeros to a power of two) is
// halved at each shuffle offset: a lane keeps one half and adds its partner's
// copy of that half, so nf values cost about nf shuffles instead of 5 nf; once
// one value is left the remaining offsets are plain butterflies.  The lane's
// offset bits then give the index of the sum it holds.
std::string gen_reduce_store(size_t nf, const std::string &acc, const std::string &dst, bool to_float)
{
    std::ostringstream os;
    size_t p2 = 1;
    while (p2 < nf) p2 <<= 1;
    std::vector<std::string> L;
    for (size_t f = 0; f < p2; ++f) L.push_back(f < nf ? "s" + std::to_string(f) : "(" + acc + ")0");
    std::string idx = "0";
    int dup = 0, tmp = 0;
    for (int o = 16; o >= 1; o >>= 1) {
        const std::string O = std::to_string(o);
        if (L.size() == 1) {
            os << "            " << L[0] << " += __shfl_xor_sync(NNP_FULL, " << L[0] << ", " << O << ");\n";
            dup |= o;
            continue;
        }
        const size_t h = L.size() / 2;
        os << "            const bool hb" << O << " = (lane & " << O << ") != 0;\n";
        std::vector<std::string> N;
        for (size_t i = 0; i < h; ++i) {
            const std::string t = "rs" + std::to_string(tmp++);
            os << "            " << acc << " " << t << " = (hb" << O << " ? " << L[h + i] << " : " << L[i]
               << ") + __shfl_xor_sync(NNP_FULL, hb" << O << " ? " << L[i] << " : " << L[h + i] << ", " << O << ");\n";
            N.push_back(t);
        }
        idx += " + (hb" + O + " ? " + std::to_string(h) + " : 0)";
        L = N;
    }
    os << "            { const int fi = " << idx << ";\n"
       << "              if ((lane & " << dup << ") == 0 && fi < " << nf << ") " << dst << "[fi] = "
       << (to_float ? "(float)" : "") << L[0] << "; }\n";
    return os.str();
}

// Body of one block's symmetry functions; written relative to the
// block's first function (Gb), so blocks with equal parameters share it.
std::string gen_symm_body(const Engine &E, const DevBlockA &B)
{
    std::ostringstream os;
    const std::vector<Fn> fs = block_fns(E, B);
    os << "        {\n";
    for (size_t f = 0; f < fs.size(); ++f) os << "            Acc s" << f << " = 0;\n";
    os << "            PairIt it = pit_init(k, lane);\n"
          "#pragma unroll 1\n"
          "            for (int p = lane; p < k.npairs; p += 32, pit_next(k, it)) {\n";
    std::ostringstream body;
    std::vector<float> bases;
    std::set<int> damps;
    pair_prologue(body, B, fs, bases, damps, false);
    Powers P(body);
    for (size_t f = 0; f < fs.size(); ++f) {
        const std::string x = P.power(base_of(bases, fs[f].lf), fs[f].zeta, fs[f].iz);
        body << "            acc_add(s" << f << ", " << x << ", P" << fs[f].damp << ");\n";
    }
    os << body.str() << "            }\n";
    os << gen_reduce_store(fs.size(), "Acc", "Gb", true);
    os << "            return true;\n        }\n";
    return os.str();
}

// Pair pass of one block (see force_pairs_generic), relative to the
// block's first dE/dG (eb); coefficients of pair (g, f) at g s + f - qoff
// (qoff: no generated local may take a parameter's name).
std::string gen_force_body(const Engine &E, const DevBlockA &B)
{
    std::ostringstream os;
    const std::vector<Fn> fs = block_fns(E, B);
    os << "        {\n";
    // dE/dG of the block and the coefficients of x^(zeta-1) in dE/dcos
    for (size_t f = 0; f < fs.size(); ++f) {
        os << "            const float e" << f << " = eb[" << f << "];\n";
        os << "            const float q" << f << " = e" << f << " * " << flit(fs[f].zeta * fs[f].lf) << ";\n";
    }
    os << "            PairIt it = pit_init(k, c0 + lane);\n"
          "#pragma unroll NNP_FORCE_UNROLL\n"
          "            for (int p = c0 + lane; p < c1; p += 32, pit_next(k, it)) {\n";
    std::ostringstream body;
    std::vector<float> bases;
    std::set<int> damps;
    pair_prologue(body, B, fs, bases, damps, true);
    Powers P(body);
    std::map<int, std::string> sc, sp;   // per damping group
    for (size_t f = 0; f < fs.size(); ++f) {
        const Fn &g = fs[f];
        const int b = base_of(bases, g.lf);
        std::string pz, pm1;
        if (g.iz >= 0) {
            pz = P.pw(b, g.iz);
            pm1 = (g.iz >= 1) ? P.pw(b, g.iz - 1) : "";
        } else {
            pm1 = P.power(b, g.zeta - 1.f, -1);
            pz = "(" + pm1 + " * x" + std::to_string(b) + ")";
        }
        if (!pm1.empty()) sc[g.damp] += (sc[g.damp].empty() ? "" : " + ") + ("q" + std::to_string(f) + " * " + pm1);
        sp[g.damp] += (sp[g.damp].empty() ? "" : " + ") + ("e" + std::to_string(f) + " * " + pz);
    }
    body << "            float hc = 0.f, hra = 0.f, hrb = 0.f;\n";
    for (int d : damps) {
        const std::string c = sc[d].empty() ? "0.f" : sc[d];
        const std::string s = sp[d].empty() ? "0.f" : sp[d];
        body << "            { const float gsc = " << c << ";\n";
        body << "              const float gsp = " << s << ";\n";
        body << "              hc = fmaf(gsc, P" << d << ", hc);\n";
        body << "              hra = fmaf(gsp, A" << d << ", hra);\n";
        body << "              hrb = fmaf(gsp, B" << d << ", hrb); }\n";
    }
    body << "            pair_coeffs(v.pc, v.pcs, it.g * k.s + it.f - qoff, hc, hra, hrb, cs, ua.w, ub.w);\n";
    os << body.str() << "            }\n            return true;\n        }\n";
    return os.str();
}

// Radial term of one neighbour in the force kernel: amp = sum_f e_f dG_f/dr,
// (rs, eta) and the form as literals, for GAUSSIAN dG_f/dr = exp(-g^2) (-2 eta
// g fc + fc'), g = eta (r - rs); relative to the block's first dE/dG (eb).
std::string gen_radial_force_body(const Engine &E, const DevBlockR &B)
{
    std::ostringstream os;
    os << "        {\n            float amp = 0.f;\n";
    for (int f = 0; f < B.n; ++f) {
        const float2 q = E.rpar_host[B.par + f];
        if (B.form != RAD_GAUSSIAN) {
            os << "            { float val, der; radial_fd(" << B.form << ", r, " << flit(q.x) << ", " << flit(q.y)
               << ", fc, fcd, val, der); amp = fmaf(eb[" << f << "], der, amp); }\n";
            continue;
        }
        os << "            { const float g = " << flit(q.y) << " * (r - " << flit(q.x) << ");\n"
           << "              amp = fmaf(eb[" << f << "], expf(-g * g) * fmaf(" << flit(-2.f * q.y)
           << " * g, fc, fcd), amp); }\n";
    }
    os << "            out = amp;\n            return true;\n        }\n";
    return os.str();
}

// One pair's values of a block's functions: acc[f] += x^zeta w[d] (w: products
// of the damping factors of the two neighbours).
std::string gen_few_symm_body(const Engine &E, const DevBlockA &B)
{
    std::ostringstream os, body;
    const std::vector<Fn> fs = block_fns(E, B);
    std::vector<float> bases;
    gen_bases(body, fs, bases);
    Powers P(body);
    for (size_t f = 0; f < fs.size(); ++f) {
        const std::string x = P.power(base_of(bases, fs[f].lf), fs[f].zeta, fs[f].iz);
        body << "            acc[" << f << "] = fmaf(" << x << ", w[" << fs[f].damp << "], acc[" << f << "]);\n";
    }
    os << "        {\n" << body.str() << "            return;\n        }\n";
    return os.str();
}

// One pair's share of the block's tangents: acc[f] += dx^zeta/dcos w[d] + x^zeta dw[d].
std::string gen_few_tangent_body(const Engine &E, const DevBlockA &B)
{
    std::ostringstream os, body;
    const std::vector<Fn> fs = block_fns(E, B);
    std::vector<float> bases;
    gen_bases(body, fs, bases);
    Powers P(body);
    for (size_t f = 0; f < fs.size(); ++f) {
        const int b = base_of(bases, fs[f].lf);
        const std::string d = std::to_string(fs[f].damp), F = std::to_string(f), pz = P.pw(b, fs[f].iz);
        body << "            acc[" << F << "] = fmaf(" << pz << ", dw[" << d << "], acc[" << F << "]);\n";
        if (fs[f].iz >= 1) {
            const std::string pm1 = P.pw(b, fs[f].iz - 1);
            body << "            acc[" << F << "] = fmaf(" << flit(fs[f].zeta * fs[f].lf) << " * " << pm1 << ", w[" << d << "], acc["
                 << F << "]);\n";
        }
    }
    os << "        {\n" << body.str() << "            return;\n        }\n";
    return os.str();
}

// Slopes of one radial block's functions at a neighbour: row[f] = dG_f/dr.
std::string gen_radial_drow_body(const Engine &E, const DevBlockR &B)
{
    std::ostringstream os;
    os << "        {\n            const float c = fc[" << B.cut << "], cd = fd[" << B.cut << "];\n";
    for (int f = 0; f < B.n; ++f) {
        const float2 q = E.rpar_host[B.par + f];
        if (B.form == RAD_GAUSSIAN)
            os << "            { const float g = " << flit(q.y) << " * (r - " << flit(q.x) << "); row[" << f
               << "] = expf(-g * g) * fmaf(" << flit(-2.f * q.y) << " * g, c, cd); }\n";
        else
            os << "            { float val; radial_fd(" << B.form << ", r, " << flit(q.x) << ", " << flit(q.y)
               << ", c, cd, val, row[" << f << "]); }\n";
    }
    os << "            return;\n        }\n";
    return os.str();
}

// One pair's dE/dcos and dE/dr of both neighbours from e = dE/dG of the block.
std::string gen_few_force_body(const Engine &E, const DevBlockA &B)
{
    std::ostringstream os, body;
    const std::vector<Fn> fs = block_fns(E, B);
    std::vector<float> bases;
    gen_bases(body, fs, bases);
    Powers P(body);
    std::set<int> damps;
    for (const Fn &f : fs) damps.insert(f.damp);
    for (int d : damps) body << "            float c" << d << " = 0.f, s" << d << " = 0.f;\n";
    for (size_t f = 0; f < fs.size(); ++f) {
        const int b = base_of(bases, fs[f].lf);
        const std::string d = std::to_string(fs[f].damp), F = std::to_string(f);
        const std::string pz = P.pw(b, fs[f].iz);
        body << "            s" << d << " = fmaf(e[" << F << "], " << pz << ", s" << d << ");\n";
        if (fs[f].iz >= 1) {
            const std::string pm1 = P.pw(b, fs[f].iz - 1);
            body << "            c" << d << " = fmaf(e[" << F << "] * " << flit(fs[f].zeta * fs[f].lf) << ", " << pm1 << ", c"
                 << d << ");\n";
        }
    }
    for (int d : damps)
        body << "            hc = fmaf(c" << d << ", wa[" << d << "] * wb[" << d << "], hc);\n"
             << "            ha = fmaf(s" << d << ", wda[" << d << "] * wb[" << d << "], ha);\n"
             << "            hb = fmaf(s" << d << ", wa[" << d << "] * wdb[" << d << "], hb);\n";
    os << "        {\n" << body.str() << "            return;\n        }\n";
    return os.str();
}

// The potential's cutoffs and, when every centre element has the same ones,
// its damping factors as literals of the moment kernels (class M of
// nnp_moments.cuh).
std::string gen_moment_constants(const Engine &E)
{
    std::ostringstream os;
    const DevPot &d = E.dpot;
    auto pick = [&](const char *type, const char *name, int n, const std::function<std::string(int)> &v) {
        os << "    __device__ static constexpr " << type << " " << name << "(int k) { return ";
        for (int k = 0; k + 1 < n; ++k) os << "k == " << k << " ? " << v(k) << " : ";
        os << v(n - 1) << "; }\n";
    };
    pick("DevCut", "cut", d.ncut, [&](int c) {
        return "DevCut{" + std::to_string(d.cut[c].name) + ", " + flit(d.cut[c].rc) + ", " + flit(d.cut[c].rci) + ", " +
               flit(d.cut[c].pirci) + "}";
    });
    pick("float", "rci_lo", d.ncut, [&](int c) { return flit((float)(1.0 / E.cut64_host[c] - (double)d.cut[c].rci)); });
    bool same = true;
    for (int II = 1; II < d.ntypes; ++II) {
        same = same && d.t[II].ndamp == d.t[0].ndamp;
        for (int k = 0; same && k < d.t[0].ndamp; ++k)
            same = d.t[II].damp_a[k] == d.t[0].damp_a[k] && d.t[II].damp_cut[k] == d.t[0].damp_cut[k] &&
                   E.mom_a_lo(II, k) == E.mom_a_lo(0, k);
    }
    os << "    static constexpr bool SAME = " << (same ? "true" : "false") << ";\n";
    pick("float", "damp_a", E.mom_ND, [&](int k) { return flit(d.t[0].damp_a[k]); });
    pick("float", "damp_lo", E.mom_ND, [&](int k) { return flit(E.mom_a_lo(0, k)); });
    pick("int", "damp_cut", E.mom_ND, [&](int k) { return std::to_string(d.t[0].damp_cut[k]); });
    pick("float", "norm", (int)E.mom_norm.size(), [&](int k) { return flit((float)E.mom_norm[k]); });
    pick("float", "gnorm", (int)E.mom_gnorm.size(), [&](int k) { return flit((float)E.mom_gnorm[k]); });
    return os.str();
}

// Values of one radial block's functions at a neighbour, (rs, eta) as
// literals: row[f] = G_f(r) with the block's cutoff value.
std::string gen_radial_row_body(const Engine &E, const DevBlockR &B)
{
    std::ostringstream os;
    os << "        {\n            const float c = fc[" << B.cut << "];\n";
    for (int f = 0; f < B.n; ++f) {
        const float2 q = E.rpar_host[B.par + f];
        if (B.form == RAD_GAUSSIAN)
            os << "            { const float g = " << flit(q.y) << " * (r - " << flit(q.x) << "); row[" << f
               << "] = expf(-g * g) * c; }\n";
        else
            os << "            { float d; radial_fd(" << B.form << ", r, " << flit(q.x) << ", " << flit(q.y)
               << ", c, 0.f, row[" << f << "], d); }\n";
    }
    os << "            return;\n        }\n";
    return os.str();
}

// Tangent of one block's symmetry functions along the displacement field
// (see tangent_body): per pair dG_f = zeta lf x^(zeta-1) P dcos
// + x^zeta (A rr_a + B rr_b), relative to the block's first
// entry of the tangent row (Cb).
std::string gen_tangent_body(const Engine &E, const DevBlockA &B)
{
    std::ostringstream os;
    const std::vector<Fn> fs = block_fns(E, B);
    os << "        {\n";
    for (size_t f = 0; f < fs.size(); ++f) os << "            float s" << f << " = 0.f;\n";
    os << "            PairIt it = pit_init(k, lane);\n"
          "#pragma unroll 1\n"
          "            for (int p = lane; p < k.npairs; p += 32, pit_next(k, it)) {\n";
    std::ostringstream body;
    std::vector<float> bases;
    std::set<int> damps;
    pair_prologue(body, B, fs, bases, damps, true);
    body << "            const float rra = v.pc[a], rrb = v.pc[b];\n"
            "            const float uba = ub.x * v.gx[a] + ub.y * v.gy[a] + ub.z * v.gz[a];\n"
            "            const float uab = ua.x * v.gx[b] + ua.y * v.gy[b] + ua.z * v.gz[b];\n"
            "            const float dcos = (uba - cs * rra) * ua.w + (uab - cs * rrb) * ub.w;\n";
    for (int d : damps) {
        body << "            const float W" << d << " = P" << d << " * dcos;\n";
        body << "            const float R" << d << " = fmaf(A" << d << ", rra, B" << d << " * rrb);\n";
    }
    Powers P(body);
    for (size_t f = 0; f < fs.size(); ++f) {
        const Fn &g = fs[f];
        const int b = base_of(bases, g.lf);
        std::string pz, pm1;
        if (g.iz >= 0) {
            pz = P.pw(b, g.iz);
            pm1 = (g.iz >= 1) ? P.pw(b, g.iz - 1) : "";
        } else {
            pm1 = P.power(b, g.zeta - 1.f, -1);
            pz = "(" + pm1 + " * x" + std::to_string(b) + ")";
        }
        const std::string d = std::to_string(g.damp);
        body << "            s" << f << " = fmaf(" << pz << ", R" << d << ", s" << f << ");\n";
        if (!pm1.empty())
            body << "            s" << f << " = fmaf(" << pm1 << ", " << flit(g.zeta * g.lf) << " * W" << d << ", s" << f
                 << ");\n";
    }
    os << body.str() << "            }\n";
    os << gen_reduce_store(fs.size(), "float", "Cb", false);
    os << "            return true;\n        }\n";
    return os.str();
}

// switch cases of a dispatcher: keys with the same body share one case
std::string group_cases(const std::vector<std::pair<int, std::string>> &cases)
{
    std::vector<std::string> bodies;
    std::vector<std::vector<int>> keys;
    for (const auto &c : cases) {
        size_t i = 0;
        while (i < bodies.size() && bodies[i] != c.second) ++i;
        if (i == bodies.size()) {
            bodies.push_back(c.second);
            keys.emplace_back();
        }
        keys[i].push_back(c.first);
    }
    std::ostringstream os;
    for (size_t i = 0; i < bodies.size(); ++i) {
        for (int k : keys[i]) os << "        case " << k << ":\n";
        os << bodies[i];
    }
    return os.str();
}

std::string make_source(const Engine &E, const TuneParams &tp, int part)
{
    std::ostringstream os;
    // Launch-bound, unroll and chunk choices, as macros at the top of the
    // source (TuneParams; defaults in nnp_engine.h, replaced by the
    // autotuner).  Resident blocks per SM the compiler budgets registers for
    // (at most 255, 128, 85, 64 registers for 1..4 blocks of NNP_WARPS warps).
    // Measured on the batched workload: 4 blocks make the symmetry-function
    // kernel 3 % faster than 3 (64 instead of 71 registers; its shared memory
    // allows 4); the force kernel is fastest unconstrained (115 registers, 2
    // blocks by its shared memory; capped at 128 registers it is 3 % slower).
    os << "#define NNP_SYMM_MINB " << tp.symm_minb << "\n#define NNP_FORCE_MINB " << tp.force_minb
       << "\n#define NNP_FORCE_UNROLL " << tp.force_unroll << "\n";
    // pairs per chunk of the force kernel; small values split the pair rows
    // between many chunks (used by a test)
    if (tp.force_chunk != NNP_PCH) os << "#define NNP_FORCE_CHUNK " << tp.force_chunk << "\n";
    os << "#include \"nnp_moments.cuh\"\nnamespace nnp {\nstruct JitBlocks {\n";
    std::vector<std::pair<int, std::string>> sy, fo, ta, ra, rr, rd, fy, ff, ft;
    int na = 1;   // angular functions of the largest block
    const int T = E.dpot.ntypes, TT = T * (T + 1) / 2;
    for (int II = 0; II < T; ++II)
        for (int J = 0; J < T; ++J) {
            const DevBlockR &B = E.dpot.t[II].br[J];
            if (B.n > 0) ra.emplace_back(II * NNP_MAX_TYPES + J, gen_radial_force_body(E, B));
            if (B.n > 0 && E.mom_ok) rr.emplace_back(II * NNP_MAX_TYPES + J, gen_radial_row_body(E, B));
            if (B.n > 0 && E.mom_ok) rd.emplace_back(II * NNP_MAX_TYPES + J, gen_radial_drow_body(E, B));
        }
    for (int II = 0; II < T; ++II)
        for (int tt = 0; tt < TT; ++tt) {
            const DevBlockA &B = E.dpot.t[II].ba[tt];
            if (B.n == 0) continue;
            na = std::max(na, B.n);
            if (E.mom_ok) {
                fy.emplace_back(II * NNP_MAX_TT + tt, gen_few_symm_body(E, B));
                ff.emplace_back(II * NNP_MAX_TT + tt, gen_few_force_body(E, B));
                ft.emplace_back(II * NNP_MAX_TT + tt, gen_few_tangent_body(E, B));
            } else {
                sy.emplace_back(II * NNP_MAX_TT + tt, gen_symm_body(E, B));
                fo.emplace_back(II * NNP_MAX_TT + tt, gen_force_body(E, B));
            }
            ta.emplace_back(II * NNP_MAX_TT + tt, gen_tangent_body(E, B));
        }
    os << "    template <typename Acc>\n"
          "    __device__ static bool symm(const NbrView &v, int II, int tt, const Blk &k, int cap, int lane, float *Gb)\n"
          "    {\n        switch (II * NNP_MAX_TT + tt) {\n"
       << group_cases(sy) << "        default: return false;\n        }\n    }\n";
    os << "    __device__ static bool force(const NbrView &v, int II, int tt, const Blk &k, int c0, int c1, int qoff,\n"
          "                                 int cap, int lane, const float *eb)\n"
          "    {\n        switch (II * NNP_MAX_TT + tt) {\n"
       << group_cases(fo) << "        default: return false;\n        }\n    }\n";
    os << "    template <class E>\n"
          "    __device__ static bool radial_force(int II, int t, float r, float fc, float fcd, E eb, float &out)\n"
          "    {\n        switch (II * NNP_MAX_TYPES + t) {\n"
       << group_cases(ra) << "        default: return false;\n        }\n    }\n";
    // radial sums of the symmetry-function kernel with the form fixed per case
    {
        bool used[16] = {};
        for (int II = 0; II < T; ++II)
            for (int J = 0; J < T; ++J) {
                const DevBlockR &B = E.dpot.t[II].br[J];
                if (B.n > 0 && B.form >= 0 && B.form < 16) used[B.form] = true;
            }
        os << "    template <typename Acc>\n"
              "    __device__ static bool radial_symm(int form, const NbrView &v, const float *fcv, float rs, float eta,\n"
              "                                       int k0, int s1, int G, Acc &acc)\n"
              "    {\n        switch (form) {\n";
        for (int f = 0; f < 16; ++f)
            if (used[f])
                os << "        case " << f << ": acc = radial_sum<" << f << ", Acc>(v, fcv, rs, eta, k0, s1, G); return true;\n";
        os << "        default: return false;\n        }\n    }\n";
        os << "    __device__ static bool radial_tangent(int form, const NbrView &v, const float *fcv, const float *fdv,\n"
              "                                          const float *rr, float rs, float eta, int k0, int s1, int G,\n"
              "                                          float &acc)\n"
              "    {\n        switch (form) {\n";
        for (int f = 0; f < 16; ++f)
            if (used[f])
                os << "        case " << f << ": acc = radial_tangent_sum<" << f
                   << ">(v, fcv, fdv, rr, rs, eta, k0, s1, G); return true;\n";
        os << "        default: return false;\n        }\n    }\n";
    }
    os << "    __device__ static bool tangent(const NbrView &v, int II, int tt, const Blk &k, int cap, int lane, float *Cb)\n"
          "    {\n        switch (II * NNP_MAX_TT + tt) {\n"
       << group_cases(ta) << "        default: return false;\n        }\n    }\n};\n";
    if (E.mom_ok)
        os << "struct JitMoments : JitBlocks {\n"
              "    static constexpr int T = " << T << ", L = " << E.mom_L << ", ND = " << E.mom_ND << ", NR = " << E.mom_NR
           << ", NA = " << na << ", NCUT = " << E.dpot.ncut << ";\n"
           << gen_moment_constants(E)
           << "    __device__ static void radial_row(int II, int t, float r, const float *fc, float *row)\n"
              "    {\n        switch (II * NNP_MAX_TYPES + t) {\n"
           << group_cases(rr) << "        default: return;\n        }\n    }\n"
              "    __device__ static void radial_drow(int II, int t, float r, const float *fc, const float *fd, float *row)\n"
              "    {\n        switch (II * NNP_MAX_TYPES + t) {\n"
           << group_cases(rd) << "        default: return;\n        }\n    }\n"
              "    __device__ static void few_tangent(int II, int tt, float cs, const float *w, const float *dw, float *acc)\n"
              "    {\n        switch (II * NNP_MAX_TT + tt) {\n"
           << group_cases(ft) << "        default: return;\n        }\n    }\n"
              "    __device__ static void few_symm(int II, int tt, float cs, const float *w, float *acc)\n"
              "    {\n        switch (II * NNP_MAX_TT + tt) {\n"
           << group_cases(fy) << "        default: return;\n        }\n    }\n"
              "    __device__ static void few_force(int II, int tt, float cs, const float *e, const float *wa, const float *wda,\n"
              "                                     const float *wb, const float *wdb, float &hc, float &ha, float &hb)\n"
              "    {\n        switch (II * NNP_MAX_TT + tt) {\n"
           << group_cases(ff) << "        default: return;\n        }\n    }\n};\n";
    os << "}  // namespace nnp\n";
    if (E.mom_ok && part == JIT_BASE)
        os << R"(
extern "C" __global__ void __launch_bounds__(NNP_MOM_SYMM_WARPS * 32, 7)
k_symm_jit(long long lo, long long hi, const nnp::DevPot *__restrict__ pot, const float *__restrict__ tab, int fmax,
   const int *__restrict__ type, const int *__restrict__ order, const float4 *__restrict__ nbr,
   const int *__restrict__ nbr_cnt, int cap, int gstride, float *__restrict__ G, float2 *mom,
   unsigned short *__restrict__ mom_cnt, const nnp::MomLists ls)
{
    extern __shared__ float4 smem4[];
    nnp::mom_symm_body<nnp::JitMoments>(lo, hi, pot, tab, fmax, type, order, nbr, nbr_cnt, cap, gstride, G, mom, mom_cnt, ls,
        reinterpret_cast<float *>(smem4));
}
)";
    if (E.mom_ok && (part == JIT_BASE || part == JIT_PAIR))
        os << R"(
#define NNP_FORCE_KERNEL(name, na, ...) \
extern "C" __global__ void __launch_bounds__(__VA_ARGS__) \
name(int nmain, long long lo, long long hi, const nnp::DevPot *__restrict__ pot, const float *__restrict__ tab, int fmax, \
     const float2 *__restrict__ rpar, const int *__restrict__ type, const int *__restrict__ order, \
     const float4 *__restrict__ nbr, const int *__restrict__ nbr_cnt, int cap, int gstride, \
     const float *__restrict__ dEdG, const float2 *__restrict__ mom, int msh, const unsigned short *__restrict__ mom_cnt, \
     const nnp::MomLists ls, double *__restrict__ F, nnp::DevErr *err, \
     const int *__restrict__ atom_struct, double *__restrict__ vir) \
{ \
    extern __shared__ float4 smem4[]; \
    const int nfew = (int)gridDim.x - nmain; \
    if ((int)blockIdx.x >= nfew) \
        nnp::mom_force_body<nnp::JitMoments, na>((int)blockIdx.x - nfew, nmain, lo, hi, pot, tab, fmax, rpar, type, order, nbr, nbr_cnt, cap, \
            gstride, dEdG, mom, msh, ls.mask, F, err, atom_struct, vir, reinterpret_cast<float *>(smem4)); \
    else if (na == 1) { \
        nnp::mom_wide_force_body<nnp::JitMoments>((int)blockIdx.x, nfew, NNP_MOM_FORCE_WARPS * 32, ls, lo, pot, tab, fmax, \
            type, order, nbr, cap, gstride, mom_cnt, dEdG, F, err, atom_struct, vir); \
        nnp::mom_few_force_body<nnp::JitMoments>((int)blockIdx.x, nfew, NNP_MOM_FORCE_WARPS * 32, ls, lo, pot, tab, fmax, \
            type, order, nbr, cap, gstride, mom_cnt, dEdG, F, err, atom_struct, vir); \
    } \
}
)";
    if (E.mom_ok && part == JIT_BASE) os << "NNP_FORCE_KERNEL(k_force_jit, 1, NNP_MOM_FORCE_WARPS * 32, 5)\n";
    if (E.mom_ok && part == JIT_PAIR)
        os << R"(
NNP_FORCE_KERNEL(k_force_jit2, 2, NNP_MOM_FORCE_WARPS * 32)
extern "C" __global__ void __launch_bounds__(NNP_MOM_FEW_THREADS, NNP_MOM_LIST_BLOCKS)
k_force_list(const nnp::MomLists ls, long long lo,
             const nnp::DevPot *__restrict__ pot, const float *__restrict__ tab, int fmax, const int *__restrict__ type,
             const int *__restrict__ order, const float4 *__restrict__ nbr, int cap, int gstride,
             const unsigned short *__restrict__ mom_cnt, const float *__restrict__ dEdG, double *__restrict__ F,
             nnp::DevErr *err, const int *__restrict__ atom_struct)
{
    nnp::mom_wide_force_body<nnp::JitMoments>((int)blockIdx.x, (int)gridDim.x, NNP_MOM_FEW_THREADS, ls, lo, pot, tab,
        fmax, type, order, nbr, cap, gstride, mom_cnt, dEdG, F, err, atom_struct, nullptr);
    nnp::mom_few_force_body<nnp::JitMoments>((int)blockIdx.x, (int)gridDim.x, NNP_MOM_FEW_THREADS, ls, lo, pot, tab,
        fmax, type, order, nbr, cap, gstride, mom_cnt, dEdG, F, err, atom_struct, nullptr);
}
)";
    if (part == JIT_SYMM_T)
        os << R"(
extern "C" __global__ void __launch_bounds__(NNP_MOM_FEW_THREADS, NNP_MOM_LIST_BLOCKS)
k_symm_list(const nnp::MomLists ls, long long lo,
     const nnp::DevPot *__restrict__ pot, const float *__restrict__ tab, int fmax, const int *__restrict__ type,
     const int *__restrict__ order, const float4 *__restrict__ nbr, int cap, int gstride,
     const unsigned short *__restrict__ mom_cnt, float *__restrict__ G)
{
    nnp::mom_list_symm_body<nnp::JitMoments>(ls, lo, pot, tab, fmax, type, order, nbr, cap, gstride, mom_cnt, G);
}
extern "C" __global__ void __launch_bounds__(NNP_MOM_THREADS, 2)
k_symm_jit_t(long long lo, long long hi, const nnp::DevPot *__restrict__ pot, const float *__restrict__ tab, int fmax,
   const int *__restrict__ type, const int *__restrict__ order, const float4 *__restrict__ nbr,
   const int *__restrict__ nbr_cnt, int cap, int gstride, float *__restrict__ G, float2 *mom,
   unsigned short *__restrict__ mom_cnt, const nnp::MomLists ls)
{
    extern __shared__ float4 smem4[];
    nnp::mom_symm_thread_body<nnp::JitMoments>(lo, hi, pot, tab, fmax, type, order, nbr, nbr_cnt, cap, gstride, G, mom, mom_cnt, ls,
        reinterpret_cast<float *>(smem4));
}
)";
    if (part == JIT_FORCE_T)
        os << R"(
extern "C" __global__ void __launch_bounds__(NNP_MOM_THREADS, 2)
k_force_jit_t(int nmain, long long lo, long long hi, const nnp::DevPot *__restrict__ pot, const float *__restrict__ tab, int fmax,
     const float2 *__restrict__ rpar, const int *__restrict__ type, const int *__restrict__ order,
     const float4 *__restrict__ nbr, const int *__restrict__ nbr_cnt, int cap, int gstride,
     const float *__restrict__ dEdG, const float2 *__restrict__ mom, const unsigned long long *__restrict__ mom_mask,
     double *__restrict__ F, nnp::DevErr *err)
{
    extern __shared__ float4 smem4[];
    nnp::mom_force_thread_body<nnp::JitMoments>((int)blockIdx.x, nmain, lo, hi, pot, tab, fmax, rpar, type, order, nbr,
        nbr_cnt, cap, gstride, dEdG, mom, mom_mask, F, err, reinterpret_cast<float *>(smem4));
}
)";
    if (part == JIT_TANGENT_T)
        os << R"(
extern "C" __global__ void __launch_bounds__(NNP_MOM_THREADS, 2)
k_tangent_jit_t(long long lo, long long hi, const nnp::DevPot *__restrict__ pot, const float *__restrict__ tab, int fmax,
     const int *__restrict__ type, const int *__restrict__ order, const float4 *__restrict__ nbr,
     const int *__restrict__ nbr_cnt, int cap, int gstride, const float4 *__restrict__ V, const float2 *__restrict__ mom,
     float2 *momd, const unsigned long long *__restrict__ mom_mask, float *__restrict__ Cout)
{
    extern __shared__ float4 smem4[];
    nnp::mom_tangent_thread_body<nnp::JitMoments>(lo, hi, pot, tab, fmax, type, order, nbr, nbr_cnt, cap, gstride, V, mom, momd,
        mom_mask, Cout, reinterpret_cast<float *>(smem4));
}
extern "C" __global__ void __launch_bounds__(NNP_MOM_FEW_THREADS, NNP_MOM_LIST_BLOCKS)
k_tangent_list(const nnp::MomLists ls, long long lo,
     const nnp::DevPot *__restrict__ pot, const float *__restrict__ tab, int fmax, const int *__restrict__ type,
     const int *__restrict__ order, const float4 *__restrict__ nbr, int cap, int gstride,
     const unsigned short *__restrict__ mom_cnt, const float4 *__restrict__ V, float *__restrict__ Cout)
{
    nnp::mom_list_tangent_body<nnp::JitMoments>(ls, lo, pot, tab, fmax, type, order, nbr, cap, gstride, mom_cnt, V, Cout);
}
)";
    if (!E.mom_ok && part == JIT_BASE)
        os << R"(
extern "C" __global__ void __launch_bounds__(NNP_WARPS * 32, NNP_SYMM_MINB)
k_symm_jit(long long N, const nnp::DevPot *__restrict__ pot, const float2 *__restrict__ rpar,
           const float4 *__restrict__ apar, const int *__restrict__ type, const int *__restrict__ order,
           const float4 *__restrict__ nbr,
           const int *__restrict__ nbr_cnt, int cap, int ncut_max, int ndamp_max, int gstride, float *__restrict__ G)
{
    extern __shared__ float4 smem4[];
    nnp::symm_body<float, nnp::JitBlocks>(N, pot, rpar, apar, type, order, nbr, nbr_cnt, cap, ncut_max, ndamp_max, gstride,
                                          G, reinterpret_cast<float *>(smem4));
}

extern "C" __global__ void __launch_bounds__(NNP_WARPS * 32, NNP_FORCE_MINB)
k_force_jit(long long N, const nnp::DevPot *__restrict__ pot, const float2 *__restrict__ rpar,
            const float4 *__restrict__ apar, const int *__restrict__ type, const int *__restrict__ order,
           const float4 *__restrict__ nbr,
            const int *__restrict__ nbr_cnt, int cap, int ncut_max, int ndamp_max, int gstride,
            const float *__restrict__ dEdG, double *__restrict__ F, nnp::DevErr *err,
            const int *__restrict__ atom_struct, double *__restrict__ vir)
{
    extern __shared__ float4 smem4[];
    nnp::force_body<nnp::JitBlocks>(N, pot, rpar, apar, type, order, nbr, nbr_cnt, cap, ncut_max, ndamp_max, gstride, dEdG,
                                    F, err, reinterpret_cast<float *>(smem4), atom_struct, vir);
}

)";
    if (part == JIT_TANGENT)
        os << R"(
extern "C" __global__ void __launch_bounds__(NNP_WARPS * 32, 1)
k_tangent_jit(long long N, const nnp::DevPot *__restrict__ pot, const float2 *__restrict__ rpar,
              const float4 *__restrict__ apar, const int *__restrict__ type, const int *__restrict__ order,
              const float4 *__restrict__ nbr, const int *__restrict__ nbr_cnt, int cap, int ncut_max, int ndamp_max,
              int gstride, const float4 *__restrict__ V, float *__restrict__ Cout)
{
    extern __shared__ float4 smem4[];
    nnp::tangent_body<nnp::JitBlocks>(N, pot, rpar, apar, type, order, nbr, nbr_cnt, cap, ncut_max, ndamp_max, gstride, V,
                                      Cout, reinterpret_cast<float *>(smem4));
}
)";
    return os.str();
}

}  // namespace

std::string jit_source(const Engine &E, const TuneParams &p) { return make_source(E, p, JIT_BASE); }

// The kernels of each part, with the handle's places for them; empty when the
// potential has none.
static std::vector<std::pair<const char *, void **>> part_kernels(Engine &E, int part)
{
    switch (part) {
    case JIT_BASE:
        if (E.mom_ok) return {{"k_symm_jit", &E.jit_symm_mom}, {"k_force_jit", &E.jit_force_mom1}};
        return {{"k_symm_jit", &E.jit_symm}, {"k_force_jit", &E.jit_force}};
    case JIT_PAIR:
        if (!E.mom_ok) return {};
        return {{"k_force_jit2", &E.jit_force_mom2}, {"k_force_list", &E.jit_force_list}};
    case JIT_SYMM_T:
        if (!E.mom_ok || !E.mom_thread()) return {};
        return {{"k_symm_jit_t", &E.jit_symm_momt}, {"k_symm_list", &E.jit_symm_list}};
    case JIT_FORCE_T:
        if (!E.mom_ok || !E.mom_force_thread()) return {};
        return {{"k_force_jit_t", &E.jit_force_momt}};
    case JIT_TANGENT:
        return {{"k_tangent_jit", &E.jit_tangent}};
    case JIT_TANGENT_T:
        if (!E.mom_ok || !E.mom_force_thread()) return {};
        return {{"k_tangent_jit_t", &E.jit_tangent_momt}, {"k_tangent_list", &E.jit_tangent_list}};
    }
    return {};
}

// Loaded libraries, shared by the process's handles of one potential: loading and
// the first launch of each kernel take ~0.5 ms per handle.  A library is unloaded
// with the last handle that uses it.
struct SharedLibrary {
    cudaLibrary_t lib;
    int users;
};
static std::mutex lib_mu;
static std::map<uint64_t, SharedLibrary> &libraries()
{
    static auto *m = new std::map<uint64_t, SharedLibrary>;   // outlives handles that are closed at exit
    return *m;
}

static std::string library_acquire(const std::string &source, const std::vector<char> &cubin, cudaLibrary_t &lib)
{
    const uint64_t key = source_hash(source);
    std::lock_guard<std::mutex> lk(lib_mu);
    auto it = libraries().find(key);
    if (it == libraries().end()) {
        if (cudaLibraryLoadData(&lib, cubin.data(), nullptr, nullptr, 0, nullptr, nullptr, 0) != cudaSuccess) {
            cudaGetLastError();
            return "cudaLibraryLoadData failed";
        }
        it = libraries().insert({key, {lib, 0}}).first;
    }
    ++it->second.users;
    lib = it->second.lib;
    return "";
}

static void library_release(cudaLibrary_t lib)
{
    std::lock_guard<std::mutex> lk(lib_mu);
    for (auto it = libraries().begin(); it != libraries().end(); ++it)
        if (it->second.lib == lib) {
            if (--it->second.users == 0) {
                cudaLibraryUnload(lib);
                libraries().erase(it);
            }
            return;
        }
}

void jit_release(Engine &E)
{
    for (int p = 0; p < JIT_PARTS; ++p) {
        if (E.jit_part[p]) library_release((cudaLibrary_t)E.jit_part[p]);
        E.jit_part[p] = nullptr;
        for (auto &f : part_kernels(E, p)) *f.second = nullptr;
    }
    E.jit_module = nullptr;
    E.jit_tried = 0;
}

std::string &jit_last_log()
{
    static thread_local std::string log;
    return log;
}

// 64-bit FNV-1a of a text: key of the compiled-kernel and tuning caches
uint64_t source_hash(const std::string &s)
{
    uint64_t h = 1469598103934665603ull;
    for (unsigned char c : s) {
        h ^= c;
        h *= 1099511628211ull;
    }
    return h;
}

// Directory of the on-disk caches: NNP_CACHE_DIR, else ~/.cache/nnp_b200
// ("" when neither is known).
std::string cache_dir()
{
    const char *dir = std::getenv("NNP_CACHE_DIR");
    if (dir && dir[0]) return dir;
    if (const char *home = std::getenv("HOME")) return std::string(home) + "/.cache/nnp_b200";
    return "";
}

std::string cache_path(uint64_t h)
{
    const std::string d = cache_dir();
    if (d.empty()) return "";
    char name[64];
    std::snprintf(name, sizeof name, "/%016llx.cubin", (unsigned long long)h);
    return d + name;
}

// Compiles a part of the specialised kernels with launch choices tp; cubins are
// kept per process and on disk (cache_dir()) by a hash of the source.  Safe to call
// from several host threads at once.
std::string jit_compile_params(const Engine &E, const TuneParams &tp, int part, std::string &source, std::vector<char> &cubin)
{
    static std::mutex mu;
    static std::map<uint64_t, std::vector<char>> memo;
    source = make_source(E, tp, part);
    const uint64_t key = source_hash(source + kDeviceHeaderSource + kMomentsHeaderSource);
    {
        std::lock_guard<std::mutex> lk(mu);
        auto it = memo.find(key);
        if (it != memo.end()) {
            cubin = it->second;
            return "";
        }
    }
    const std::string path = cache_path(key);
    if (!path.empty()) {
        std::ifstream in(path, std::ios::binary);
        if (in) {
            std::vector<char> buf((std::istreambuf_iterator<char>(in)), std::istreambuf_iterator<char>());
            if (!buf.empty()) {
                cubin = buf;
                std::lock_guard<std::mutex> lk(mu);
                memo[key] = buf;
                return "";
            }
        }
    }
    nvrtcProgram prog;
    const char *hdr_src[2] = {kDeviceHeaderSource, kMomentsHeaderSource};
    const char *hdr_name[2] = {"nnp_device.cuh", "nnp_moments.cuh"};
    if (nvrtcCreateProgram(&prog, source.c_str(), "nnp_jit.cu", 2, hdr_src, hdr_name) != NVRTC_SUCCESS)
        return "nvrtcCreateProgram failed";
    const char *opts[] = {"--gpu-architecture=sm_100a", "-std=c++17", "--fmad=true",
                          "--ptxas-options=-v"};
    const nvrtcResult rc = nvrtcCompileProgram(prog, 4, opts);
    size_t logn = 0;
    nvrtcGetProgramLogSize(prog, &logn);
    std::string log(logn, '\0');
    if (logn) nvrtcGetProgramLog(prog, &log[0]);
    while (!log.empty() && log.back() == '\0') log.pop_back();   // the size counts the terminator
    if (rc != NVRTC_SUCCESS) {
        nvrtcDestroyProgram(&prog);
        return "run-time compilation failed: " + log.substr(0, 2000);
    }
    jit_last_log() = log;
    size_t n = 0;
    nvrtcGetCUBINSize(prog, &n);
    cubin.resize(n);
    nvrtcGetCUBIN(prog, cubin.data());
    nvrtcDestroyProgram(&prog);
    {
        std::lock_guard<std::mutex> lk(mu);
        memo[key] = cubin;
    }
    if (!path.empty()) {
        const std::string dir = path.substr(0, path.rfind('/'));
        std::string cmd;
        for (size_t k = 1; k <= dir.size(); ++k)
            if (k == dir.size() || dir[k] == '/') mkdir(dir.substr(0, k).c_str(), 0755);
        const std::string tmp = path + ".tmp" + std::to_string((long long)getpid());
        std::ofstream out(tmp, std::ios::binary);
        if (out) {
            out.write(cubin.data(), (std::streamsize)cubin.size());
            out.close();
            std::rename(tmp.c_str(), path.c_str());
        }
    }
    return "";
}

// Compiles every part in `parts` that the potential has, side by side: NVRTC takes
// seconds for each, and the call waits for the longest.
static std::vector<std::string> compile_parts(const Engine &E, const std::vector<int> &parts, std::vector<std::string> &src,
                                              std::vector<std::vector<char>> &cubin, std::vector<std::string> &log)
{
    const size_t n = parts.size();
    std::vector<std::string> msg(n);
    src.resize(n);
    cubin.resize(n);
    log.resize(n);
    auto one = [&](size_t k) {
        jit_last_log().clear();
        msg[k] = jit_compile_params(E, E.tune, parts[k], src[k], cubin[k]);
        log[k] = jit_last_log();
    };
    std::vector<std::thread> th;
    for (size_t k = 1; k < n; ++k) {
        try {
            th.emplace_back(one, k);
        } catch (const std::system_error &) {        // no thread to be had
            one(k);
        }
    }
    if (n) one(0);
    for (auto &t : th) t.join();
    return msg;
}

std::string jit_check(Engine &E, std::string &log)
{
    std::vector<int> parts;
    for (int p = 0; p < JIT_PARTS; ++p)
        if (!part_kernels(E, p).empty()) parts.push_back(p);
    std::vector<std::string> src, logs;
    std::vector<std::vector<char>> cubin;
    const std::vector<std::string> msg = compile_parts(E, parts, src, cubin, logs);
    for (size_t k = 0; k < parts.size(); ++k) {
        if (!msg[k].empty()) return msg[k];
        log += logs[k] + "\n" + src[k];
    }
    return "";
}

// Loads the parts of the bit set `want` that the handle has not loaded yet.  A part
// that fails is not tried again: its kernels stay null, and the calls take the other
// ones.  Not while a stream is captured (the eager call before has them loaded).
std::string jit_need(Engine &E, unsigned want)
{
    want &= ~E.jit_tried;
    if (!want) return "";
    E.jit_tried |= want;
    std::vector<int> parts;
    for (int p = 0; p < JIT_PARTS; ++p)
        if ((want >> p & 1) && !part_kernels(E, p).empty()) parts.push_back(p);
    std::vector<std::string> src, log;
    std::vector<std::vector<char>> cubin;
    std::vector<std::string> msg = compile_parts(E, parts, src, cubin, log);
    std::string first;
    for (size_t k = 0; k < parts.size(); ++k) {
        cudaLibrary_t lib = nullptr;
        if (msg[k].empty()) msg[k] = library_acquire(src[k], cubin[k], lib);
        if (msg[k].empty()) {
            E.jit_part[parts[k]] = (void *)lib;
            if (parts[k] == JIT_BASE) E.jit_source = src[k];
            for (auto &f : part_kernels(E, parts[k])) {
                cudaKernel_t q;
                if (cudaLibraryGetKernel(&q, lib, f.first) != cudaSuccess) {
                    cudaGetLastError();
                    msg[k] = "run-time kernels not found";
                    break;
                }
                *f.second = (void *)q;
                cudaFuncSetAttribute((const void *)q, cudaFuncAttributeMaxDynamicSharedMemorySize, NNP_SMEM_MAX);
                if (std::getenv("NNP_JIT_VERBOSE")) {    // registers and local memory of the compiled kernels
                    cudaFuncAttributes a;
                    if (cudaFuncGetAttributes(&a, (const void *)q) == cudaSuccess)
                        std::fprintf(stderr, "nnp jit: %s %d registers, %zu bytes local memory\n", f.first, a.numRegs,
                                     a.localSizeBytes);
                    else
                        cudaGetLastError();
                }
            }
            if (!msg[k].empty())
                for (auto &f : part_kernels(E, parts[k])) *f.second = nullptr;
        }
        if (first.empty()) first = msg[k];
    }
    return first;
}

std::string jit_build(Engine &E)
{
    jit_release(E);
    const std::string msg = jit_need(E, 1u << JIT_BASE);
    if (!msg.empty()) {
        jit_release(E);
        return msg;
    }
    E.jit_module = E.jit_part[JIT_BASE];
    return "";
}

std::string jit_launch(void *fn, int grid, int block, size_t smem, cudaStream_t stream, void **args)
{
    const void *k = (const void *)fn;
    const cudaError_t r = cudaLaunchKernel(k, dim3(grid), dim3(block), args, smem, stream);
    if (r != cudaSuccess) return std::string("cudaLaunchKernel: ") + cudaGetErrorString(r);
    return "";
}

}  // namespace nnp
