// Host planning for the radiality kernels: configuration (INI), ring
// deduplication and per-axis factorisation, separable Catmull-Rom weight
// tables, interpolation windows and block lists.
#include <algorithm>
#include <array>
#include <cctype>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <tuple>
#include <vector>

#include "srrf_internal.h"

namespace rfba {

// ---------------------------------------------------------------------------
// Configuration

// GradientCalc.cpp:19-41 defaults.
void config_default(rfba_srrf_config* c) {
    c->ring_radius = 0.5f;
    c->mag[0] = c->mag[1] = c->mag[2] = 5;
    c->axes_in_ring = 6;
    c->main_range = 1;
    c->x_range = c->y_range = c->z_range = 0;
    c->method = 1;
    c->itc = 1;
    c->trac_order = 2;
    c->remove_con = 0;
    c->renormalize = 0;
    c->gradient_smooth = 0;
    c->intensity_w = 1;
    c->block_size[0] = c->block_size[1] = c->block_size[2] = 16;
}

namespace {
std::string trim(const std::string& s) {
    size_t a = 0, b = s.size();
    while (a < b && std::isspace((unsigned char)s[a])) ++a;
    while (b > a && std::isspace((unsigned char)s[b - 1])) --b;
    return s.substr(a, b - a);
}
bool ieq(const std::string& a, const std::string& b) {
    if (a.size() != b.size()) return false;
    for (size_t i = 0; i < a.size(); ++i)
        if (std::tolower((unsigned char)a[i]) != std::tolower((unsigned char)b[i])) return false;
    return true;
}
}  // namespace

// Profile-file reader with the lookup rules the reference relies on
// (GetPrivateProfileString/Int, GradientCalc.cpp:15-42): section and key
// names are case-insensitive, the first matching key wins, a missing file,
// section or key gives the default, integers parse like atoi.
struct Ini {
    std::vector<std::tuple<std::string, std::string, std::string>> kv;
    bool load(const char* path) {
        FILE* f = std::fopen(path, "r");
        if (!f) return false;
        char line[2048];
        std::string sec;
        while (std::fgets(line, sizeof line, f)) {
            std::string l = trim(line);
            if (l.empty() || l[0] == ';') continue;
            if (l[0] == '[') {
                size_t e = l.find(']');
                sec = trim(l.substr(1, e == std::string::npos ? std::string::npos : e - 1));
                continue;
            }
            size_t eq = l.find('=');
            if (eq == std::string::npos) continue;
            std::string v = trim(l.substr(eq + 1));
            if (v.size() >= 2 && v.front() == '"' && v.back() == '"') v = v.substr(1, v.size() - 2);
            kv.emplace_back(sec, trim(l.substr(0, eq)), v);
        }
        std::fclose(f);
        return true;
    }
    const std::string* find(const char* sec, const char* key) const {
        for (auto& e : kv)
            if (ieq(std::get<0>(e), sec) && ieq(std::get<1>(e), key)) return &std::get<2>(e);
        return nullptr;
    }
    int geti(const char* sec, const char* key, int def) const {
        const std::string* v = find(sec, key);
        return v ? std::atoi(v->c_str()) : def;
    }
    float getf(const char* sec, const char* key, float def) const {
        const std::string* v = find(sec, key);
        return v ? (float)std::atof(v->c_str()) : def;
    }
};

bool config_load_ini(const char* path, rfba_srrf_config* c) {
    config_default(c);
    Ini ini;
    bool ok = ini.load(path);
    c->ring_radius = ini.getf("SRRF", "RingRadius", 0.5f);
    int m = ini.geti("SRRF", "Magnification", 5);
    c->mag[0] = c->mag[1] = c->mag[2] = m;
    c->axes_in_ring = ini.geti("SRRF", "AxesinRing", 6);
    c->main_range = ini.geti("SRRF", "MainRange", 1);
    c->x_range = ini.geti("SRRF", "XRange", 0);
    c->y_range = ini.geti("SRRF", "YRange", 0);
    c->z_range = ini.geti("SRRF", "ZRange", 0);
    c->method = ini.geti("Temproal", "Method", 1);
    c->itc = ini.geti("Temproal", "Integrate_Temporal_Correlations", 1);
    c->trac_order = ini.geti("Temproal", "TRAC_ORDER", 2);
    c->remove_con = ini.geti("Radiality", "Remove_Positivity_Constraint", 0);
    c->renormalize = ini.geti("Radiality", "Renormalize", 0);
    c->gradient_smooth = ini.geti("Radiality", "Gradient_Smoothing", 0);
    c->intensity_w = ini.geti("Weighting", "Intensity_Weighting", 1);
    c->block_size[0] = ini.geti("Split", "BlockSizeX", 16);
    c->block_size[1] = ini.geti("Split", "BlockSizeY", 16);
    c->block_size[2] = ini.geti("Split", "BlockSizeZ", 16);
    return ok;
}

bool config_validate(const rfba_srrf_config& c, std::string* err) {
    char buf[256];
    for (int a = 0; a < 3; ++a)
        if (c.mag[a] < 1 || c.mag[a] > kMaxMag) {
            std::snprintf(buf, sizeof buf, "magnification %d on axis %d outside [1, %d]", c.mag[a], a, kMaxMag);
            *err = buf;
            return false;
        }
    if (!(c.ring_radius > 0.f) || !std::isfinite(c.ring_radius)) {
        *err = "ring radius must be a positive number";
        return false;
    }
    if (c.axes_in_ring < 1 || c.axes_in_ring > 32) {
        *err = "AxesinRing must be in [1, 32]";
        return false;
    }
    const int rs[4] = {c.main_range, c.x_range, c.y_range, c.z_range};
    for (int r : rs)
        if (r < 0 || r > kMaxGradRange) {
            std::snprintf(buf, sizeof buf, "gradient ranges must be in [0, %d]", kMaxGradRange);
            *err = buf;
            return false;
        }
    if (c.method < 0 || c.method > 3) {
        *err = "Method must be 0 (TRM), 1 (TRA), 2 (TRPPM) or 3 (TRAC)";
        return false;
    }
    if (c.method == 3 && (c.trac_order < 2 || c.trac_order > 4)) {
        *err = "TRAC_ORDER must be 2, 3 or 4";
        return false;
    }
    return true;
}

// ---------------------------------------------------------------------------
// Ring

// kernel.cu:17 and :23-33: float angle step (PI = 3.141592654f), float sin/cos,
// (r * sin) * cos association.
static void raw_ring(float r, int n, std::vector<float>& x, std::vector<float>& y, std::vector<float>& z) {
    x.resize(n * n);
    y.resize(n * n);
    z.resize(n * n);
    const float step = (3.141592654f * 2.0f) / (float)n;
    for (int i = 0; i < n; ++i)
        for (int j = 0; j < n; ++j) {
            const int k = i * n + j;
            x[k] = r * std::sin(step * (float)i) * std::cos(step * (float)j);
            y[k] = r * std::sin(step * (float)i) * std::sin(step * (float)j);
            z[k] = r * std::cos(step * (float)i);
        }
}

static int value_index(std::vector<float>& vals, float v, float tol) {
    for (size_t i = 0; i < vals.size(); ++i)
        if (std::fabs(vals[i] - v) <= tol) return (int)i;
    vals.push_back(v);
    return (int)vals.size() - 1;
}

// Distinct points of the ring and their multiplicities. Points that coincide up
// to float rounding of sin/cos (|d| <= 1e-6 r) are one point; coordinates within
// 1e-6 r of 0 are 0.
static void distinct_points(float r, const std::vector<float>& rx, const std::vector<float>& ry,
                            const std::vector<float>& rz, std::vector<std::array<float, 3>>* reps,
                            std::vector<int>* mult) {
    const float tol = 1e-6f * r;
    auto snap = [&](float v) { return std::fabs(v) <= tol ? 0.f : v; };
    for (size_t i = 0; i < rx.size(); ++i) {
        const float px = snap(rx[i]), py = snap(ry[i]), pz = snap(rz[i]);
        int found = -1;
        for (size_t k = 0; k < reps->size(); ++k)
            if (std::fabs((*reps)[k][0] - px) <= tol && std::fabs((*reps)[k][1] - py) <= tol &&
                std::fabs((*reps)[k][2] - pz) <= tol) {
                found = (int)k;
                break;
            }
        if (found < 0) {
            reps->push_back({px, py, pz});
            mult->push_back(1);
        } else
            (*mult)[found]++;
    }
}

bool build_ring_plan(const rfba_srrf_config& c, RingPlan* rp, std::string* err) {
    const int n = 2 * c.axes_in_ring;
    const float r = c.ring_radius;
    rp->n = n;
    raw_ring(r, n, rp->rx, rp->ry, rp->rz);
    rp->npoints_raw = n * n;
    const float tol = 1e-6f * r;
    std::vector<std::array<float, 3>> reps;
    std::vector<int> mult;
    distinct_points(r, rp->rx, rp->ry, rp->rz, &reps, &mult);
    // distinct axis values, sorted
    std::vector<float> xv, yv, zv;
    for (auto& p : reps) {
        value_index(xv, p[0], tol);
        value_index(yv, p[1], tol);
        value_index(zv, p[2], tol);
    }
    std::sort(xv.begin(), xv.end());
    std::sort(yv.begin(), yv.end());
    std::sort(zv.begin(), zv.end());
    struct P {
        int a, b, c;
    };
    std::vector<P> pts;
    for (auto& p : reps) pts.push_back({value_index(xv, p[0], tol), value_index(yv, p[1], tol), value_index(zv, p[2], tol)});
    std::sort(pts.begin(), pts.end(), [](const P& u, const P& v) {
        return std::tie(u.a, u.b, u.c) < std::tie(v.a, v.b, v.c);
    });
    rp->xv = xv;
    rp->yv = yv;
    rp->zv = zv;
    rp->grp_xval.clear();
    rp->grp.clear();
    rp->pair_yval.clear();
    rp->pair_pt.clear();
    rp->pt_zval.clear();
    rp->zero_x = rp->zero_y = -1;
    for (size_t i = 0; i < xv.size(); ++i)
        if (xv[i] == 0.f) rp->zero_x = (int)i;
    for (size_t i = 0; i < yv.size(); ++i)
        if (yv[i] == 0.f) rp->zero_y = (int)i;
    if (rp->zero_x < 0 || rp->zero_y < 0) {
        *err = "ring has no point on the z axis";
        return false;
    }
    int last_a = -1, last_b = -1;
    for (size_t k = 0; k < pts.size(); ++k) {
        const P& p = pts[k];
        if (p.a != last_a) {
            rp->grp_xval.push_back(p.a);
            rp->grp.push_back((int)rp->pair_yval.size());
            last_a = p.a;
            last_b = -1;
        }
        if (p.b != last_b) {
            rp->pair_yval.push_back(p.b);
            rp->pair_pt.push_back((int)k);
            last_b = p.b;
        }
        rp->pt_zval.push_back(p.c);
    }
    rp->grp.push_back((int)rp->pair_yval.size());
    rp->pair_pt.push_back((int)pts.size());
    return true;
}

int ring_zero_pair(const RingPlan& rp) {
    for (size_t g = 0; g + 1 < rp.grp.size(); ++g) {
        if (rp.grp_xval[g] != rp.zero_x) continue;
        for (int p = rp.grp[g]; p < rp.grp[g + 1]; ++p)
            if (rp.pair_yval[p] == rp.zero_y) return p;
    }
    return -1;
}

// ---------------------------------------------------------------------------
// Tap weights

// Catmull-Rom kernel, a = 0.5 (kernel.cu:128-138), evaluated in double.
static double cubic(double xx) {
    const double a = 0.5;
    double x = std::fabs(xx);
    if (x < 1.0) return x * x * (x * (-a + 2.0) + (a - 3.0)) + 1.0;
    if (x < 2.0) return -a * x * x * x + 5.0 * a * x * x - 8.0 * a * x + 4.0 * a;
    return 0.0;
}

// For fine index X = mag*xi + ph and ring offset rho, the sample sits at
// q = xi + f with f = (ph + 0.5 + rho) / mag; the reference's taps are
// u0-1..u0+2 with u0 = floor(q - 0.5) (kernel.cu:149-166). With f in
// [-0.5, 1.5) the taps lie in xi-2..xi+2: 4 of them start at xi-2+off,
// off = floor(f - 0.5) + 1.
static bool tap4(int ph, double rho, int mag, float w[4], int* off) {
    const double f = (ph + 0.5 + rho) / mag;
    if (!(f >= -0.5 && f < 1.5)) return false;
    const int u0 = (int)std::floor(f - 0.5);
    *off = u0 + 1;
    for (int k = 0; k < 4; ++k) w[k] = (float)cubic(f - ((u0 - 1 + k) + 0.5));
    return true;
}
static bool tap5(int ph, double rho, int mag, float w[5]) {
    const double f = (ph + 0.5 + rho) / mag;
    if (!(f >= -0.5 && f < 1.5)) return false;
    for (int m = 0; m < 5; ++m) w[m] = (float)cubic(f - ((m - 2) + 0.5));
    return true;
}

// ---------------------------------------------------------------------------
// Forward plan

bool build_forward_plan(const rfba_srrf_config& c, FwdPlan* fp, std::string* err) {
    const int n = 2 * c.axes_in_ring;
    const float r = c.ring_radius, tol = 1e-6f * r;
    std::vector<float> raw[3];
    raw_ring(r, n, raw[0], raw[1], raw[2]);
    std::vector<std::array<float, 3>> reps;
    std::vector<int> mult;
    distinct_points(r, raw[0], raw[1], raw[2], &reps, &mult);
    struct P {
        int a, b, c, m;
        double u[3];
    };
    // one order of the axes: distinct values, points grouped by mid and then x
    // value, and the pairs' start indices
    struct Order {
        std::vector<float> val[3];
        std::vector<P> pts;
        std::vector<int> pair0;
    };
    auto arrange = [&](int a1, int a2) {
        Order o;
        const int ax[3] = {0, a1, a2};
        for (int k = 0; k < 3; ++k) {
            for (auto& p : reps) value_index(o.val[k], p[ax[k]], tol);
            value_index(o.val[k], 0.f, tol);  // the intensity's sample
            std::sort(o.val[k].begin(), o.val[k].end());
        }
        for (size_t i = 0; i < reps.size(); ++i) {
            P p;
            p.a = value_index(o.val[0], reps[i][0], tol);
            p.b = value_index(o.val[1], reps[i][a1], tol);
            p.c = value_index(o.val[2], reps[i][a2], tol);
            p.m = mult[i];
            for (int k = 0; k < 3; ++k) p.u[k] = (double)reps[i][ax[k]] / r;
            o.pts.push_back(p);
        }
        // nearest the centre first, +v and -v next to each other: samples on opposite
        // sides mostly cancel, so the running sum stays small (in value order its
        // rounding made the map's error against 64 bits a fifth larger)
        std::vector<int> rank[2];
        for (int k = 0; k < 2; ++k) {
            std::vector<float> mag;
            for (float v : o.val[k]) value_index(mag, std::fabs(v), tol);
            std::sort(mag.begin(), mag.end());
            for (float v : o.val[k]) rank[k].push_back(value_index(mag, std::fabs(v), tol));
        }
        std::sort(o.pts.begin(), o.pts.end(), [&](const P& u, const P& v) {
            return std::make_tuple(rank[1][u.b], u.b, rank[0][u.a], u.a, u.c) <
                   std::make_tuple(rank[1][v.b], v.b, rank[0][v.a], v.a, v.c);
        });
        for (size_t i = 0; i < o.pts.size(); ++i) {
            const P& p = o.pts[i];
            const bool axis = p.u[0] == 0 && p.u[1] == 0;
            if (i == 0 || axis || p.a != o.pts[i - 1].a || p.b != o.pts[i - 1].b) o.pair0.push_back((int)i);
        }
        return o;
    };
    // clocks per subvoxel up to a common factor: 22 a pair's second pass, 7 a
    // group's first (as in forward_depth)
    auto cost = [&](const Order& o, int a2) {
        int groups = 0;
        for (size_t i = 0; i < o.pts.size(); ++i) groups += i == 0 || o.pts[i].b != o.pts[i - 1].b;
        return (22.0 * o.pair0.size() + 7.0 * groups) / c.mag[a2];
    };
    Order o = arrange(1, 2);
    fp->ax1 = 1;
    fp->ax2 = 2;
    {
        Order alt = arrange(2, 1);
        if (cost(alt, 1) < cost(o, 2)) {
            o = std::move(alt);
            fp->ax1 = 2;
            fp->ax2 = 1;
        }
    }
    const int ax[3] = {0, fp->ax1, fp->ax2};
    for (int k = 0; k < 3; ++k) fp->mag[k] = c.mag[ax[k]];

    // lane tables
    std::vector<float>& L = fp->lane;
    L.clear();
    auto bits = [](int v) {
        float f;
        std::memcpy(&f, &v, 4);
        return f;
    };
    static const char* const names = "xyz";
    auto too_large = [&](int axis) {
        *err = std::string("ring radius too large for the ") + names[axis] +
               " magnification (needs ring_radius < (1 + mag)/2)";
        return false;
    };
    // taps of one value at every phase; the offsets as a mask
    auto taps = [&](int k, float v, std::vector<std::array<float, 4>>* w, std::vector<int>* off) {
        for (int ph = 0; ph < fp->mag[k]; ++ph) {
            std::array<float, 4> t;
            int of;
            if (!tap4(ph, v, fp->mag[k], t.data(), &of)) return too_large(ax[k]);
            w->push_back(t);
            off->push_back(of);
        }
        return true;
    };
    int* wpos[2] = {&fp->l_wx, &fp->l_wm};
    int* opos[2] = {&fp->l_offx, &fp->l_offm};
    std::vector<std::array<float, 4>> w, w_x;
    std::vector<int> off, x_mask;
    for (int k = 0; k < 2; ++k) {
        w.clear();
        off.clear();
        for (float v : o.val[k])
            if (!taps(k, v, &w, &off)) return false;
        *wpos[k] = (int)L.size();
        for (auto& t : w) L.insert(L.end(), t.begin(), t.end());
        if (k == 0) {
            w_x = w;
            for (size_t i = 0; i < off.size(); ++i) {
                if (i % fp->mag[0] == 0) x_mask.push_back(0);
                x_mask.back() |= off[i] << (i % fp->mag[0]);
            }
        }
        *opos[k] = (int)L.size();
        for (int of : off) L.push_back(bits(of));
        while (L.size() % 4) L.push_back(0.f);
    }
    fp->zero_x = value_index(o.val[0], 0.f, tol);
    fp->zero_m = value_index(o.val[1], 0.f, tol);
    fp->zero_xoff = x_mask[fp->zero_x];

    // uniform tables
    const int mz = fp->mag[2];
    const int npairs = (int)o.pair0.size(), npts = (int)o.pts.size(), nzv = (int)o.val[2].size();
    std::vector<std::array<int, 3>> groups;
    for (int i = 0; i < npairs; ++i) {
        const int b = o.pts[o.pair0[i]].b;
        if (groups.empty() || groups.back()[0] != b) groups.push_back({b, i, i});
        groups.back()[2] = i + 1;
    }
    fp->ngroups = (int)groups.size();
    fp->npairs = npairs;
    fp->npoints = npts;
    fp->u_grp = 0;
    fp->u_pair = fp->ngroups;
    fp->u_pt = fp->u_pair + 4 * npairs;
    fp->u_wz = fp->u_pt + 3 * npts;
    fp->u_wi = fp->u_wz + 2 * nzv * mz;
    std::vector<float>& U = fp->utab;
    U.clear();
    auto put = [&](double a, double b, double cc, double d) {
        for (double v : {a, b, cc, d}) U.push_back((float)v);
    };
    auto put_bits = [&](int a, int b, int cc, int d) {
        for (int v : {a, b, cc, d}) U.push_back(bits(v));
    };
    for (auto& g : groups) put_bits(g[0], g[1], g[2], 0);
    // the commonest multiplicity carries the weight 1
    std::map<int, int> count;
    for (auto& p : o.pts) count[p.m]++;
    int common = o.pts[0].m;
    for (auto& e : count)
        if (e.second > count[common]) common = e.first;
    fp->neg_weight = -((float)common / (float)n);  // kernel.cu:244 divides by n, not n^2
    std::vector<double> kappa(npts, 0.0);
    for (int i = 0; i < npairs; ++i) {
        const int q0 = o.pair0[i], q1 = i + 1 < npairs ? o.pair0[i + 1] : npts;
        const P& f = o.pts[q0];
        const double ux = f.u[0], um = f.u[1];
        double pa = 1, pb = 0, ea = 0, eb = 1, scale = 1;
        int plane[3] = {2, 1, 0};
        if (ux == 0 && um == 0) {
            pa = f.u[2] < 0 ? -1 : 1;
        } else {
            plane[0] = 0;
            plane[2] = 2;
            const double h = std::sqrt(ux * ux + um * um);
            double mean = 0;
            for (int q = q0; q < q1; ++q) {
                kappa[q] = o.pts[q].u[2] / h;
                mean += std::fabs(kappa[q]) / (q1 - q0);
            }
            scale = std::sqrt(1 + mean * mean);
            pa = ux / h;
            pb = um / h;
            ea = -scale * um / h;
            eb = scale * ux / h;
        }
        put(pa, pa, pb, pb);
        put(ea, ea, eb, eb);
        put_bits(plane[0], plane[1], plane[2], f.a);
        put_bits(q0, q1, x_mask[f.a], 0);
        U.back() = (float)(kGuard * scale * scale * scale * scale);
    }
    w.clear();
    off.clear();
    for (float v : o.val[2])
        if (!taps(2, v, &w, &off)) return false;
    for (int q = 0; q < npts; ++q) {
        const P& p = o.pts[q];
        const double un = std::sqrt(p.u[0] * p.u[0] + p.u[1] * p.u[1] + p.u[2] * p.u[2]);
        const double rho = std::sqrt((double)p.m / common);
        int mask = 0;
        for (int ph = 0; ph < mz; ++ph) mask |= off[p.c * mz + ph] << ph;
        put(kappa[q], kappa[q], -kappa[q], -kappa[q]);
        put(-rho * un, -rho * un, rho, rho);
        put_bits(p.c * mz, mask, 0, 0);
    }
    for (auto& t : w) {
        put(t[0], t[0], t[1], t[1]);
        put(t[2], t[2], t[3], t[3]);
    }
    for (int ph = 0; ph < mz; ++ph) {
        float t[5];
        tap5(ph, 0.0, mz, t);
        const int m0 = 2 * ph + 1 >= mz ? 1 : 0;
        put(t[m0], t[m0 + 1], t[m0 + 2], t[m0 + 3]);
    }
    fp->adj_utab = U;
    for (int q = 0; q < npts; ++q) {
        const P& p = o.pts[q];
        const double un = std::sqrt(p.u[0] * p.u[0] + p.u[1] * p.u[1] + p.u[2] * p.u[2]);
        const double f = 2.0 * p.m / n * un;
        float* r = &fp->adj_utab[4 * (fp->u_pt + 3 * q + 1)];
        r[0] = r[1] = (float)(-f * un);
        r[2] = r[3] = (float)f;
    }
    fp->u_wx = (int)(fp->adj_utab.size() / 4);
    for (auto& t : w_x)
        for (int k : {0, 0, 1, 1, 2, 2, 3, 3}) fp->adj_utab.push_back(t[k]);
    int tile_axis[3];  // of x, y, z
    for (int k = 0; k < 3; ++k) tile_axis[ax[k]] = k;
    fp->fix.clear();
    for (int q = 0; q < npts; ++q) {
        const P& p = o.pts[q];
        const double ux = p.u[tile_axis[0]], uy = p.u[tile_axis[1]], uz = p.u[tile_axis[2]];
        const double h = std::sqrt(ux * ux + uy * uy), un = std::sqrt(ux * ux + uy * uy + uz * uz);
        for (double v : {h > 0 ? ux / h : 1.0, h > 0 ? uy / h : 0.0, h / un, uz / un}) fp->fix.push_back((float)v);
        for (float v : {(float)p.m / (float)n * (2.0f * (float)un), (float)un,
                        (float)std::sqrt(1 + kappa[q] * kappa[q]), 0.f})
            fp->fix.push_back(v);
    }
    return true;
}

FwdParams forward_params(const FwdPlan& fp, const rfba_srrf_config& c, const void* in, int in_u16, const int dims[4],
                         int ty, int cz) {
    FwdParams p;
    std::memset(&p, 0, sizeof p);
    p.in = in;
    p.in_u16 = in_u16;
    p.W = dims[0];
    p.H = dims[1];
    p.D = dims[2];
    p.T = dims[3];
    for (int a = 0; a < 3; ++a) p.mag[a] = fp.mag[a];
    p.ax1 = fp.ax1;
    p.ax2 = fp.ax2;
    const int lat[3] = {c.x_range, c.y_range, c.z_range};
    p.gr[0] = c.gradient_smooth == 0 ? 1 : c.main_range;
    p.gr[1] = c.gradient_smooth == 0 ? 0 : lat[0];
    p.gr[2] = c.gradient_smooth == 0 ? 0 : lat[fp.ax1];
    p.gr[3] = c.gradient_smooth == 0 ? 0 : lat[fp.ax2];
    p.R = std::max(std::max(p.gr[0], p.gr[1]), std::max(p.gr[2], p.gr[3]));
    const auto ranges = [&](int a, int b) { return p.gr[0] == a && p.gr[1] == b && p.gr[2] == b && p.gr[3] == b; };
    p.grad_mode = ranges(1, 1) ? 1 : ranges(1, 0) ? 2 : 0;
    p.TY = ty > 0 ? ty : kTileRows;
    p.cz = cz;
    p.NU = (kTileX - 1) / fp.mag[0] + 2 + 4;
    p.NV = (p.TY - 1) / fp.mag[1] + 2 + 4;
    p.NIX = p.NU + 2 * p.R;
    p.NIY = p.NV + 2 * p.R;
    p.NIZ = 4 * tile_quads(cz) + 2 * p.R;
    p.u_region = radiality_u_region(p);
    p.renorm = c.renormalize == 1;
    p.poscon = c.remove_con == 1;
    p.lane_words = (int)fp.lane.size();
    p.l_wx = fp.l_wx;
    p.l_offx = fp.l_offx;
    p.l_wm = fp.l_wm;
    p.l_offm = fp.l_offm;
    p.u_count = (int)(fp.utab.size() / 4);
    p.u_grp = fp.u_grp;
    p.u_pair = fp.u_pair;
    p.u_pt = fp.u_pt;
    p.u_wz = fp.u_wz;
    p.u_wi = fp.u_wi;
    p.ngroups = fp.ngroups;
    p.zero_x = fp.zero_x;
    p.zero_m = fp.zero_m;
    p.zero_xoff = fp.zero_xoff;
    p.u_wx = fp.u_wx;
    p.neg_weight = fp.neg_weight;
    p.tma_bx = radiality_tma_box_x(p);
    return p;
}

FwdParams adjoint_params(const FwdPlan& fp, const rfba_srrf_config& c, const void* in, const int dims[4], int cz) {
    FwdParams p = forward_params(fp, c, in, 0, dims, 0, cz);
    p.tma_bx = 0;
    p.u_region = radiality_adjoint_u_region(p);
    p.u_count = (int)(fp.adj_utab.size() / 4);
    return p;
}

// (tile, volume) pairs of tiles of cz cells and kTileRows rows; tiles: their number along
// the innermost axis, over the regions
static long long tile_items(const FwdPlan& fp, const std::vector<FwdRegion>& regions, int T, int cz, double* tiles) {
    const int mz = fp.mag[2], fz = mz * cz;
    long long items = 0;
    for (auto& r : regions) {
        const int lo = r.lo[fp.ax2], hi = r.hi[fp.ax2];
        const int n = (hi - (lo / mz) * mz + fz - 1) / fz;
        if (tiles) *tiles += n;
        items += (long long)n * ((r.hi[0] - r.lo[0] + kTileX - 1) / kTileX) *
                 ((r.hi[fp.ax1] - r.lo[fp.ax1] + kTileRows - 1) / kTileRows) * T;
    }
    return items;
}

int forward_depth(const FwdPlan& fp, const std::vector<FwdRegion>& regions, int T, int sms) {
    // Two items or fewer to an SM: a launch lasts as long as one item, and a shallower one
    // ends sooner. 5 x 10x12x12 at mag 2, the whole call: 63.6 us with 8 cells, 55.5 with
    // 4. At innermost magnifications from kFlatMag on 4 cells are 20 to 32 subvoxels deep
    // already, and 2 are left: 5x6x8 at mag 6 and 5 axes 86 us with 4 cells, 71 with 2, 8
    // such volumes (192 items) 97 and 82, 12 of them (288) 110 and 112.
    const auto few = [&](int cz) { return tile_items(fp, regions, T, cz, nullptr) <= 2LL * sms; };
    const int shallow = fp.mag[2] >= kFlatMag && few(4) ? 2 : 4;
    if (fp.mag[2] > kDeepMag || few(8)) return shallow;
    // time per tile column in clocks (one SM, as measured): a point at one subvoxel
    // 29, a pair's second pass at one cell 22, a group's first pass at one cell 7. The
    // same holds for tables in global memory: 20 volumes of 32^3 at 2 x 2 x 2 and 16 axes
    // take 3.82 ms with shallow tiles, 3.13 with deep ones (24^3 at 4 x 4 x 2: 4.65, 4.56)
    const auto time = [&](int cz) {
        double tiles = 0;
        tile_items(fp, regions, T, cz, &tiles);
        return tiles * (fp.mag[2] * cz * 29.0 * fp.npoints + (cz + 4) * (22.0 * fp.npairs + 7.0 * fp.ngroups));
    };
    return time(4) < time(8) ? shallow : 8;
}

int adjoint_depth(const FwdPlan& fp, const FwdRegion& region, int T, int sms) {
    // Half the depth for one item or fewer to an SM. Map and derivative of 9x16x16 at mag
    // 2: one volume (12 items) 263 us with 8 cells, 223 with 4, 12 of them 279 and 251, 24
    // 338 and 389; 4x4x6 at mag 8: 417 us with 4 cells, 343 with 2. Not built for tables in
    // global memory, which are no small calls.
    const int cz = adj_cz(fp.mag[2]);
    if (fp.adj_utab.size() / 4 > (size_t)kUTabMax) return cz;
    return tile_items(fp, {region}, T, cz, nullptr) <= sms ? cz / 2 : cz;
}

void forward_tiles(const FwdPlan& fp, int ty, BlockDev* b) {
    const int rows = ty > 0 ? ty : kTileRows;
    const int mz = fp.mag[2], fz = mz * b->cz;
    b->ntile[0] = (b->nreg[0] + kTileX - 1) / kTileX;
    b->ntile[fp.ax1] = (b->nreg[fp.ax1] + rows - 1) / rows;
    b->ntile[fp.ax2] = (b->hi[fp.ax2] - (b->lo[fp.ax2] / mz) * mz + fz - 1) / fz;
}

// ---------------------------------------------------------------------------
// Windows

// The reference's sample window (kernel.cu:143-147 / 260-265) in float.
static inline bool window_ok(float x0f, int mag, int dim) {
    const float q = x0f / (float)mag;
    return !(q < 1.5f || q > (float)dim - 1.5f);
}

// Fine indices X in [0, dim*mag) whose ring samples on this axis all pass the
// window. Float addition and division are monotone, so testing the smallest and
// largest ring coordinate is exact. Returns lo > hi when none passes.
bool window_range(float, const std::vector<float>& rc, int mag, int dim, int* lo, int* hi) {
    float rmin = rc[0], rmax = rc[0];
    for (float v : rc) {
        rmin = std::min(rmin, v);
        rmax = std::max(rmax, v);
    }
    *lo = 1;
    *hi = 0;
    bool any = false;
    for (int X = 0; X < dim * mag; ++X) {
        const float xc = (float)X + 0.5f;
        if (window_ok(xc + rmin, mag, dim) && window_ok(xc + rmax, mag, dim)) {
            if (!any) *lo = X;
            *hi = X;
            any = true;
        }
    }
    return any;
}

// Fine indices whose centre passes the window (interpolateIntensity).
int fine_window_int(int mag, int dim, int* lo, int* hi) {
    *lo = 1;
    *hi = 0;
    bool any = false;
    for (int X = 0; X < dim * mag; ++X)
        if (window_ok((float)X + 0.5f, mag, dim)) {
            if (!any) *lo = X;
            *hi = X;
            any = true;
        }
    return any ? 1 : 0;
}

// ---------------------------------------------------------------------------
// Block lists

// GradientCalc.cpp:47-116 with border 2. Each block computes only the part of
// its interior that the reference's put-back leaves in the output (later
// blocks overwrite the overlap of earlier ones), so every output voxel is
// written once with the value the reference ends up with.
int blocks_gradientcalc(const rfba_srrf_config& c, const int dims[4], rfba_block* out, int cap, std::string* err) {
    const int border = 2;
    // the reference has one magnification; the extended configuration's
    // per-axis factors apply axis by axis (equal factors give the reference's blocks)
    const int* mag = c.mag;
    int split[3];
    for (int a = 0; a < 3; ++a) {
        const int step = c.block_size[a] - 2 * border;
        if (step <= 0) {
            *err = "block size must exceed 4 (GradientCalc border 2 on both sides)";
            return RFBA_ERR_INVALID;
        }
        const int num = dims[a] - 2 * border;
        split[a] = num / step;  // C truncation, as the reference
        if (num % step != 0) split[a] += 1;
        if (split[a] < 0) split[a] = 0;
    }
    const long long W = (long long)dims[0] * mag[0], H = (long long)dims[1] * mag[1];
    int count = 0;
    for (int k = 0; k < split[2]; ++k)
        for (int j = 0; j < split[1]; ++j)
            for (int i = 0; i < split[0]; ++i) {
                const int pos[3] = {i, j, k};
                rfba_block b;
                std::memset(&b, 0, sizeof b);
                bool empty = false;
                for (int a = 0; a < 3; ++a) {
                    const int step = c.block_size[a] - 2 * border;
                    const bool last = pos[a] == split[a] - 1;
                    const int res = last ? dims[a] - (split[a] - 1) * step : c.block_size[a];
                    const int start = pos[a] == 0 ? 0 : pos[a] * step;
                    b.origin[a] = start;
                    b.size[a] = res;
                    b.lo[a] = border * mag[a];
                    b.hi[a] = last ? res * mag[a] : (step + border) * mag[a];
                    if (b.hi[a] > res * mag[a]) b.hi[a] = res * mag[a];
                    if (b.hi[a] <= b.lo[a]) empty = true;
                }
                if (empty) continue;
                b.out_stride[0] = 1;
                b.out_stride[1] = W;
                b.out_stride[2] = W * H;
                b.out_offset = ((long long)b.origin[2] * mag[2] + b.lo[2]) * W * H +
                               ((long long)b.origin[1] * mag[1] + b.lo[1]) * W +
                               ((long long)b.origin[0] * mag[0] + b.lo[0]);
                if (out && count < cap) out[count] = b;
                ++count;
            }
    return count;
}

// Matlab Scripts/doSplit.m:1-19 (1-based positions turned 0-based).
static std::vector<std::pair<int, int>> dosplit_axis(int xall, int maxX, int border) {
    std::vector<std::pair<int, int>> pos;  // (start, size), 1-based start
    if (maxX >= xall) {
        pos.push_back({1, xall});
        return pos;
    }
    pos.push_back({1, maxX});
    while (pos.back().first + maxX <= xall) {
        const int nxt = pos.back().first + pos.back().second - 2 * border;
        pos.push_back({nxt, maxX});
    }
    pos.back().second = xall - pos.back().first + 1;
    return pos;
}

int blocks_dosplit(const rfba_srrf_config& c, const int dims[4], const int max_size[3], int border, rfba_block* out,
                   int cap, long long* out_elems, std::string* err) {
    if (border < 0 || max_size[0] <= 2 * border || max_size[1] <= 2 * border || max_size[2] <= 2 * border) {
        *err = "doSplit needs max size > 2*border";
        return RFBA_ERR_INVALID;
    }
    auto xs = dosplit_axis(dims[0], max_size[0], border);
    auto ys = dosplit_axis(dims[1], max_size[1], border);
    auto zs = dosplit_axis(dims[2], max_size[2], border);
    int count = 0;
    long long off = 0;
    // GenerateBlock.m:118-120 loop order: x outermost, z innermost.
    for (auto& px : xs)
        for (auto& py : ys)
            for (auto& pz : zs) {
                rfba_block b;
                std::memset(&b, 0, sizeof b);
                b.origin[0] = px.first - 1;
                b.origin[1] = py.first - 1;
                b.origin[2] = pz.first - 1;
                b.size[0] = px.second;
                b.size[1] = py.second;
                b.size[2] = pz.second;
                for (int a = 0; a < 3; ++a) {
                    b.lo[a] = 0;
                    b.hi[a] = b.size[a] * c.mag[a];
                }
                b.out_offset = off;
                b.out_stride[0] = 1;
                b.out_stride[1] = b.hi[0];
                b.out_stride[2] = (long long)b.hi[0] * b.hi[1];
                off += (long long)b.hi[0] * b.hi[1] * b.hi[2];
                if (out && count < cap) out[count] = b;
                ++count;
            }
    if (out_elems) *out_elems = off;
    return count;
}

}  // namespace rfba
