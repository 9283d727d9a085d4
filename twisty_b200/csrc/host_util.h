// host_util.h -- host-side pieces of the runner that need no device: config parsing,
// initial-curve construction, geometry checks, the closed-form normaliser.
#pragma once
#include <cstdint>
#include <map>
#include <memory>
#include <string>
#include <vector>

#include "../../include/twisty_b200.h"

namespace twisty {

// A tiny document model shared by the JSON and YAML readers.
struct Node {
    enum Kind { Null, Bool, Number, String, Object, Array } kind = Null;
    bool b = false;
    double num = 0.0;
    std::string str;
    std::map<std::string, Node> obj;
    std::vector<Node> arr;
    const Node *get(const std::string &k) const;
};

bool parse_json(const std::string &text, Node &out, std::string &err);
bool parse_yaml(const std::string &text, Node &out, std::string &err);

// Fill params/bc from a parsed config (reference schema: experiment.experimentParams.*,
// experiment.basicExperiment.*). Returns false with err set when a required key is
// missing or has the wrong type.
bool params_from_node(const Node &root, twisty_params &p, twisty_bc *bc, std::string &err);

// CalculateMinimumArclength (Twisty/PathGeneration.cpp:12-43).
float min_arclength(const twisty_bc &bc, uint32_t n);

// Initial curve for any N >= 4: points 0, 1, N-1, N fixed by the boundary conditions
// (Twisty/Curve.cpp:20-30), the N-2 free segments laid on a planar circular arc from
// point 1 to point N-1 whose turning angle is solved by bisection so that every segment
// has length exactly ds (computed in double, stored in float). The arc's plane is turned
// about the chord by an angle drawn from the bootstrap seed. Returns false (err set) when
// |x_{N-1} - x_1| > (N-2) ds.
bool bootstrap_arc(const twisty_bc &bc, uint32_t n, uint32_t seed, std::vector<float> &pos, std::string &err);

// The reference's recursive bootstrapper (Twisty/PathGeneration.cpp:47-414 from the call at
// FullExperimentRunnerOptimalPerturb.cpp:122-131) for N with N-2 in {4, 6, 8, 12, 16, 24, 32,
// 48, ...}: the same random stream and arithmetic, the reference's curve for the same
// bootstrapSeed. Returns false (err set) for other N or when the placement fails.
bool bootstrap_resolvable(uint32_t n);
bool bootstrap_reference(const twisty_bc &bc, uint32_t n, uint32_t seed, std::vector<float> &pos, std::string &err);
// kind 0: the reference bootstrapper where it resolves N, else the arc; 1: the reference's
// only; 2: the arc.
bool bootstrap_curve(const twisty_bc &bc, uint32_t n, uint32_t seed, int kind, std::vector<float> &pos, std::string &err);

// The reference's table, rounding for rounding: WeightLookupTableIntegral ctor + Initialize
// (Twisty/PathWeightUtils.cpp:281-348) with Integrate's sorted sum (:371-433) and the float
// phase function (:19-33), on host threads. Bins whose integral cancels to a tiny fraction
// of its terms keep the reference's summation-order rounding only this way, so the
// faithful table mode (the drop-in's bit-parity setup) is built here; the FP64 tables are
// built on the device. out[bins]; minmax = {min, max} weight. Returns false on bad params.
bool lut_faithful_host(float mu, float eps, float scatter, float min_bound, float max_bound, float bias,
                       uint32_t num_steps_int, uint32_t bins, float ds, float *out, float minmax[2]);

// K4 (Twisty/PathWeightUtils.cpp:643-651) and the z of Norm (:729-732), float math.
double norm_k4_log10(float z, float ds);
float norm_z(const twisty_bc &bc, float ds);

}  // namespace twisty
