"""The host side of the objective calls (objective.cpp) against a stand-in for
the CUDA runtime: device memory is a byte count with a limit, launches and
copies are counted and looked over for null pointers.  No GPU: what a call does
when an allocation fails is decided on the host."""
import json
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HOST = os.path.join(ROOT, "dugksfoam_gb300", "csrc", "host")
OK, OOM = 0, 7

DRIVER = r"""
#include <cstdio>
#include <cstring>
#include <iostream>
#include <map>
#include <memory>
#include <sstream>
#include <string>
#include <vector>
#include <atomic>
#include <mutex>
#include <functional>
#define private public
#include "objective.h"
#undef private
#include "../cuda/gradient.h"

static std::map<char*, size_t> held;
static size_t used = 0, limit = size_t(1) << 40, refuse0 = 1, refuse1 = 0;
static char* next = reinterpret_cast<char*>(size_t(1) << 44);
static char* const kMesh = reinterpret_cast<char*>(size_t(1) << 45);  // the handle's own arrays
static long launches = 0, passes = 0, nulls = 0, mallocs = 0, wild = 0;
static void see(const void* p, size_t n = 1) {  // bytes p .. p + n - 1 of one allocation
    const char* c = static_cast<const char*>(p);
    if (c < reinterpret_cast<char*>(size_t(1) << 44)) { ++nulls; return; }
    if (c >= kMesh && c + n <= kMesh + 4096) return;
    auto it = held.upper_bound(const_cast<char*>(c));
    if (it == held.begin() || (--it, c + n > it->first + it->second)) ++wild;
}

extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) {
    ++mallocs;
    if (used + n > limit || (n >= refuse0 && n <= refuse1)) return cudaErrorMemoryAllocation;
    *p = next;
    held[next] = n;
    next += n + 4096;
    used += n;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    auto it = held.find(static_cast<char*>(p));
    if (it == held.end()) return cudaErrorInvalidValue;
    used -= it->second;
    held.erase(it);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int, size_t n, cudaStream_t) { see(p, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) {
    if (k == cudaMemcpyDeviceToHost) std::memset(d, 0, n);
    else see(d, n);
    if (k != cudaMemcpyHostToDevice) see(s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) { return cudaMemcpyAsync(d, s, n, k, nullptr); }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) { *f = limit - used; *t = limit; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
}

namespace dugks {
class FusedPipeline {};
Solver::~Solver() = default;
int Solver::fail(int code, const std::string& m) { err_ = m; return code; }
int Solver::checkCuda(cudaError_t, const char*) { return 0; }
int Solver::synchronize() { return 0; }
StepArgs Solver::argsNow() const { return base_; }
void launch_ref_pass(int, const StepArgs& a, const RefBuffers& b, int, cudaStream_t) {
    ++launches; ++passes;
    for (const void* p : {(void*)b.gT, (void*)b.hT, (void*)b.gS, (void*)b.hS, (void*)b.Gbg, (void*)a.rho}) see(p);
}
void launch_ref_init(const StepArgs&, double* g, double* h, int, cudaStream_t) { ++launches; see(g); see(h); }
void launch_objective(const StepArgs&, const double*, const double*, double, double* J, cudaStream_t) { ++launches; see(J); }
void adj_pack_macros(int, const double* r, const double*, const double*, const double*, const double*, double* o, int,
                     cudaStream_t) { ++launches; see(r); see(o); }
void adj_launch_step(const AdjState& s, const double* g, const double* h, const double* m, bool, double, int, cudaStream_t) {
    ++launches;
    for (const void* p : {(void*)s.gT, (void*)s.hT, (void*)s.gS, (void*)s.hS, (void*)s.lgN, (void*)s.lhG, (void*)s.lTw,
                          (void*)g, (void*)h, (void*)m}) see(p);
}
size_t adj_table_bytes(int, int) { return 0; }
void adj_sum(int, const double* x, double* o, cudaStream_t) { ++launches; see(x); see(o); }
void tlm_launch_incabs(const TlmState& s, cudaStream_t) { ++launches; see(s.incAbs); }
void tlm_launch_init(const TlmState& s, const double*, const double*, const double*, int, cudaStream_t) {
    ++launches; see(s.gT); see(s.hT);
}
void tlm_launch_step(const TlmState& s, bool, const double*, const double*, double, Dual* J, int, cudaStream_t) {
    ++launches; see(s.gS); see(s.hG); see(J);
}

// 4 cells in a row, 64 velocities
std::unique_ptr<Solver> handle() {
    std::unique_ptr<Solver> s(new Solver());
    Mesh& m = s->mesh_;
    m.nC = 4; m.nW = 10; m.nI = 3; m.D = 2;
    m.Sf.assign(3 * 13, 1.0);
    for (int w = 0; w < 10; ++w) { m.wallFace.push_back(3 + w); m.wallPatch.push_back(0); m.wallKind.push_back(DUGKS_PATCH_MAXWELL); }
    StepArgs& a = s->base_;
    a.nC = 4; a.nI = 3; a.nW = 10; a.nA = 13; a.nV = a.Vp = 64; a.M = 8; a.D = 2; a.hasH = 1; a.muRef = 1.0;
    s->initRho_ = s->initU_ = s->initT_ = reinterpret_cast<double*>(kMesh);
    a.Tw = reinterpret_cast<double*>(kMesh);
    s->dt_ = 1.0;
    return s;
}
}  // namespace dugks

int main() {
    std::map<std::string, std::unique_ptr<dugks::Solver>> hs;
    std::string line;
    while (std::getline(std::cin, line)) {
        std::istringstream in(line);
        std::string name, what;
        in >> name >> what;
        if (name == "refuse") { refuse0 = std::stoull(what); in >> refuse1; continue; }
        if (name == "limit") { limit = std::stoull(what); continue; }
        if (what == "close") { hs.erase(name); }
        else if (!hs.count(name)) hs[name] = dugks::handle();
        int n = 1, k = 1, rc = 0;
        in >> n >> k;
        launches = passes = nulls = mallocs = wild = 0;
        dugks::Objective o;
        o.nSteps = n; o.ckptEvery = k; o.qPatch = 0;
        double J = 0, dJ = 0;
        std::vector<double> tw(10);
        if (what == "value") rc = dugks::objective_value(*hs[name], o, J);
        if (what == "tangent") rc = dugks::objective_tangent(*hs[name], o, tw.data(), 0.0, J, dJ);
        if (what == "adjoint") rc = dugks::objective_adjoint(*hs[name], o, J, tw.data(), dJ);
        std::printf("{\"rc\": %d, \"launches\": %ld, \"passes\": %ld, \"nulls\": %ld, \"mallocs\": %ld, \"wild\": %ld, \"used\": %zu}\n",
                    rc, launches, passes, nulls, mallocs, wild, used);
    }
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    """run(*lines) -> one dict per line that names a handle."""
    from dugksfoam_gb300 import build

    if shutil.which("g++") is None:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("objective")
    (d / "driver.cpp").write_text(DRIVER)
    cuda = os.path.join(os.path.dirname(os.path.dirname(build._nvcc())), "include")
    srcs = [os.path.join(HOST, f) for f in ("objective.cpp", "workspace.cpp") if os.path.exists(os.path.join(HOST, f))]
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "include"), "-I", cuda, "-I", HOST,
                    str(d / "driver.cpp"), *srcs, "-o", str(d / "driver"), "-lpthread"], check=True)

    def f(*lines):
        r = subprocess.run([str(d / "driver")], input="\n".join(lines) + "\n", capture_output=True, text=True,
                           timeout=120, check=True)
        return [json.loads(x) for x in r.stdout.splitlines()]

    return f


MB = 1 << 20
# bytes of one stored state (g~, h~, G_b of g and h, nine macros per cell) and of one step's forward values
STATE = 8 * (2 * 4 * 64 + 2 * 10 * 64 + 9 * 4)
INTER = 8 * (2 * 13 * 64 + 9 * 13 + 10)


@pytest.mark.parametrize("n, k", [(20000, 20000), (20000, 1)], ids=["segment", "checkpoints"])
def test_states_that_do_not_fit_are_refused(run, n, k):
    assert n * STATE > 80 * MB
    (r,) = run("limit %d" % (80 * MB), "a adjoint %d %d" % (n, k))
    assert r["rc"] == OOM and r["launches"] == 0 and r["nulls"] == 0


def test_face_values_that_do_not_fit_are_recomputed(run):
    n = 8000
    r, = run("a adjoint %d %d" % (n, n))
    assert r["rc"] == OK and r["nulls"] == 0 and r["passes"] == 8 * n
    # too large for half of what is free; or asked for and refused
    for line in ("limit %d" % (64 * MB + n * STATE + n * INTER // 2),
                 "refuse %d %d" % (n * INTER, n * INTER + 4096)):
        r, = run(line, "a adjoint %d %d" % (n, n))
        assert r["rc"] == OK and r["nulls"] == 0 and r["passes"] == (8 + 5) * n


@pytest.mark.parametrize("k", [1, 3, 7, 8, 2**31 - 8, 2**31 - 1])
def test_any_checkpoint_interval(run, k):
    # 7 steps: the last segment is stored as it runs, the others run twice
    r, = run("a adjoint 7 %d" % k)
    assert r["rc"] == OK and r["nulls"] == 0 and r["wild"] == 0
    assert r["passes"] == 8 * (7 + 7 - (7 - (7 - 1) // k * k))


@pytest.mark.parametrize("call", ["value 3", "tangent 3", "adjoint 3 2"])
def test_every_refused_buffer_is_an_error(run, call):
    # one allocation per buffer (no chunk of 64 MB fits): each limit ends at another one
    lines, n = [], 6000
    for i in range(n):
        lines += ["limit %d" % (256 * i), "h%d %s" % (i, call), "h%d close" % i]
    r = run(*lines)[::2]
    assert r[0]["rc"] == OOM and r[-1]["rc"] == OK
    for x in r:
        assert x["nulls"] == x["wild"] == 0 and (x["rc"] == OK or (x["rc"] == OOM and x["launches"] == 0)), x


CALLS = ["value 5", "tangent 5", "adjoint 12 12", "adjoint 8000 8000", "adjoint 8000 90", "adjoint 12000 4000"]


def _least(run, call):
    """The least device memory that a new handle needs for a call (to 1 MB)."""
    lo, hi = 0, 1024
    while hi - lo > 1:
        mid = (lo + hi) // 2
        ok = run("limit %d" % (mid * MB), "a " + call)[0]["rc"] == OK
        lo, hi = (lo, mid) if ok else (mid, hi)
    return hi * MB


@pytest.mark.parametrize("first", CALLS)
def test_a_call_fits_after_any_other_where_it_fits_alone(run, first):
    for call in CALLS:
        need = max(_least(run, call), _least(run, first))
        a, b = run("limit %d" % need, "a " + first, "a " + call)
        alone, = run("limit %d" % need, "a " + call)
        assert a["rc"] == b["rc"] == alone["rc"] == OK, (first, call, need)
        assert b["nulls"] == b["wild"] == 0 and b["used"] <= need


def test_face_values_are_stored_again_by_the_same_call(run):
    # half of what is free holds the face values, as long as kept chunks of the
    # call before count as free: every limit takes the form it took the first time
    n = 6000
    forms = set()
    for limit in range(150, 420, 10):
        a, b, c = run("limit %d" % (limit * MB), *["a adjoint %d %d" % (n, n)] * 3)
        assert a["rc"] == b["rc"] == c["rc"] == OK
        assert a["passes"] == b["passes"] == c["passes"], limit
        forms.add(a["passes"])
    assert forms == {8 * n, 13 * n}


def test_handles_keep_a_bounded_amount_together(run):
    # 3 GB a call: the kept chunks of all handles stay within 4 GiB and go with their handles
    n = 110000
    r = run(*["h%d adjoint %d %d" % (i, n, n) for i in range(4)], *["h%d close" % i for i in range(4)])
    assert all(x["rc"] == OK for x in r[:4]) and 2 << 30 < r[0]["used"]
    assert max(x["used"] for x in r) <= 4 << 30
    assert r[-1]["used"] == 0


@pytest.mark.parametrize("first", CALLS)
def test_a_call_fits_beside_idle_handles(run, first):
    for call in CALLS:
        limit = max(_least(run, call), _least(run, first))
        alone, = run("limit %d" % limit, "a " + call)
        a, b = run("limit %d" % limit, "a " + first, "b " + call)
        assert a["rc"] == b["rc"] == OK and b["nulls"] == b["wild"] == 0, (first, call)
        assert b["passes"] == alone["passes"], (first, call)
