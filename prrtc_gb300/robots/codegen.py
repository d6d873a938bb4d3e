"""Robot-model compiler: JSON collision models -> C tables + CUDA checkers.

Input: ``prrtc_gb300/robots/<robot>.json`` (written by ``extract.py``).
Output, for each robot:

* ``csrc/robots/<robot>_model.h``: the model as plain-C tables
  (``prrtc_joint_def`` ... from ``model_types.h``), read by the CPU oracle and
  by host code;
* ``csrc/robots/<robot>_fkcc.cuh``: the CUDA checker for one configuration
  per thread, in two forms.  The fast form (``near_check_*``) marks, in
  straight-line code, the groups that can possibly collide (bounds from the
  environment's clearance grid and from gate distances); only marked groups
  are walked, and where the answer is within rounding of contact the exact
  form decides.  The exact form visits the model's groups in the reference's
  order.  Joint transforms are folded at generation time (zero and unit
  entries of the fixed transforms vanish).  Also here: the joint rows of the
  clearance's kinematics (``clr_rows``).  The per-leaf work runs
  in three small shared routines supplied by the caller (``Ctx``), so code
  size stays proportional to the number of groups, not of sphere pairs:

  - ``ctx.env_hit(x, y, z, r)``: sphere against every obstacle;
  - ``ctx.env_leaves(T, leaves, n)``: leaf spheres given in frame T;
  - ``ctx.self_pairs(Tab, pairs, n)``: sphere pairs (a in frame A, b in
    frame B) given the relative transform Tab = inv(T_A) T_B;
  - ``ctx.pair_hit(dx, dy, dz, ra + rb)``: gate pair overlap test;
  - ``ctx.stop()``: cooperative early exit (another lane already failed).

Usage: ``python -m prrtc_gb300.robots.codegen`` (no reference checkout needed).
"""
from __future__ import annotations

import json
from pathlib import Path

import numpy as np

HERE = Path(__file__).resolve().parent
CSRC = HERE.parent / "csrc" / "robots"
ROBOTS = ("sphere", "panda", "fetch", "baxter")
INLINE_LEAVES = 6   # leaf blocks up to this size are emitted as straight-line tests
# Robots whose exact form is emitted in table form: every frame computed first,
# then one loop over the group schedule (run_schedule in device_common.cuh).
# Baxter's 388 groups as straight-line code overflow the instruction cache
# (its planner kernel stalled on instruction fetch 33 times per issue).
TABLE_ROBOTS = ("panda", "fetch", "baxter")
# Robots that also get the straight-line exact form, as fkcc_validate_exact.
# Which form decides single configurations within rounding of contact is part
# of their verdicts (the two are contracted differently), so it stays as it
# was chosen when the exact form made every check: 2^20 random configurations,
# Panda straight-line 1.24 ms, table 1.32; Fetch 5.38 against 5.28; Baxter's
# straight-line form does not fit the instruction cache.
INLINE_VALIDATE = ("sphere", "panda")


def load_model(robot: str) -> dict:
    return json.loads((HERE / f"{robot}.json").read_text())


def _lit(x: float) -> str:
    x = float(x)
    if x == int(x) and abs(x) < 1e6:
        return f"{x:.1f}f"
    return f"{x!r}f"


# ------------------------------------------------------------------ C tables

def emit_c_tables(m: dict) -> str:
    R = m["robot"].capitalize()
    out = []
    w = out.append
    w(f"// pRRTC {m['robot']} collision model as plain-C tables.  Generated by")
    w("// prrtc_gb300/robots/codegen.py from the fitted model; do not edit.")
    w(f"// Max |sphere centre - reference float64 FK|: {m['max_err']:.3e} m")
    w("#pragma once")
    w('#include "model_types.h"')
    w("")
    ne, ns = len(m["env_groups"]), len(m["self_groups"])
    nl = sum(len(g["leaves"]) for g in m["env_groups"])
    npairs = sum(len(g["pairs"]) for g in m["self_groups"])
    w("enum {")
    w(f"    k{R}Dof = {m['dof']},")
    w(f"    k{R}NumJoints = {len(m['joints'])},")
    w(f"    k{R}NumSpheres = {len(m['spheres'])},")
    w(f"    k{R}NumEnvGroups = {ne},")
    w(f"    k{R}NumEnvLeaves = {nl},")
    w(f"    k{R}NumSelfGroups = {ns},")
    w(f"    k{R}NumSelfPairs = {npairs},")
    w(f"    k{R}NumSchedule = {len(m['schedule'])},")
    w("};")
    w("")
    w(f"static const prrtc_joint_def k{R}Joints[] = {{")
    for jt in m["joints"]:
        F = [x for row in jt["F"] for x in row]
        w("    {%d, %d, %d, {%s}}," % (jt["q"], jt["parent"], 1 if jt["type"] == "revolute" else 0,
                                     ", ".join(_lit(x) for x in F)))
    w("};")
    w(f"static const prrtc_sphere_def k{R}Spheres[] = {{")
    for s in m["spheres"]:
        w("    {%d, %s, %s, %s, %s}," % (s["frame"], *[_lit(x) for x in s["c"]], _lit(s["r"])))
    w("};")
    w(f"static const prrtc_group_def k{R}EnvGroups[] = {{")
    off = 0
    for g in m["env_groups"]:
        w("    {%d, -1, %d, %d},  /* %s */" % (g["gate"], off, len(g["leaves"]), g["label"]))
        off += len(g["leaves"])
    w("};")
    allv = [x for g in m["env_groups"] for x in g["leaves"]]
    w(f"static const short k{R}EnvLeaves[] = {{")
    for i in range(0, len(allv), 16):
        w("    " + ", ".join(str(x) for x in allv[i:i + 16]) + ",")
    w("};")
    if ns:
        w(f"static const prrtc_group_def k{R}SelfGroups[] = {{")
        off = 0
        for g in m["self_groups"]:
            w("    {%d, %d, %d, %d},  /* %s */" % (g["gate"][0], g["gate"][1], off, len(g["pairs"]), g["label"]))
            off += len(g["pairs"])
        w("};")
        allp = [p for g in m["self_groups"] for p in g["pairs"]]
        w(f"static const short k{R}SelfPairs[][2] = {{")
        for i in range(0, len(allp), 8):
            w("    " + " ".join("{%d, %d}," % tuple(p) for p in allp[i:i + 8]))
        w("};")
    else:
        w(f"static const prrtc_group_def k{R}SelfGroups[] = {{{{-1, -1, 0, 0}}}};")
        w(f"static const short k{R}SelfPairs[][2] = {{{{0, 0}}}};")
    w(f"static const prrtc_sched_def k{R}Schedule[] = {{")
    for i in range(0, len(m["schedule"]), 8):
        w("    " + " ".join("{%d, %d}," % (0 if k == "env" else 1, g) for k, g in m["schedule"][i:i + 8]))
    w("};")
    w("")
    return "\n".join(out)


# ------------------------------------------------------- symbolic scalar code

class _Code:
    """Straight-line float code with constant folding of 0 / +-1 / literals."""

    def __init__(self):
        self.lines = []
        self.n = 0

    def tmp(self, expr, prefix="v"):
        if isinstance(expr, float):
            return expr
        name = f"{prefix}{self.n}"
        self.n += 1
        self.lines.append(f"const float {name} = {expr};")
        return name

    @staticmethod
    def term(coef: float, var):
        """coef * var as (sign, text) or a folded constant."""
        if isinstance(var, float):
            return coef * var
        if coef == 0.0:
            return 0.0
        if coef == 1.0:
            return var
        if coef == -1.0:
            return f"(-{var})"
        return f"{_lit(coef)} * {var}"

    @staticmethod
    def dot(pairs, const=0.0):
        """sum(coef * var) + const; coef may be a float or a variable name,
        var may be a variable name or a float."""
        c = float(const)
        terms = []
        for a, b in pairs:
            if isinstance(a, float) and isinstance(b, float):
                c += a * b
            elif isinstance(a, float) or isinstance(b, float):
                k, v = (a, b) if isinstance(a, float) else (b, a)
                if k == 0.0:
                    continue
                terms.append(_Code.term(k, v))
            else:
                terms.append(f"{a} * {b}")
        if not terms:
            return c
        s = terms[0]
        for t in terms[1:]:
            if t.startswith("(-"):
                s = f"{s} - {t[2:-1]}"
            else:
                s = f"{s} + {t}"
        if c != 0.0:
            s = f"{s} + {_lit(c)}" if c > 0 else f"{s} - {_lit(-c)}"
        return s


def _mat_of(F):
    return [[float(F[i][k]) for k in range(4)] for i in range(3)]


class _FkGen:
    """Emits frame computations lazily, in chain order, into a _Code."""

    def __init__(self, model, code: _Code):
        self.m = model
        self.code = code
        self.frames = {-1: [[1.0, 0.0, 0.0, 0.0], [0.0, 1.0, 0.0, 0.0], [0.0, 0.0, 1.0, 0.0]]}
        self.joint = {jt["q"]: jt for jt in model["joints"]}

    def frame(self, j):
        if j in self.frames:
            return self.frames[j]
        jt = self.joint[j]
        P = self.frame(jt["parent"])
        F = _mat_of(jt["F"])
        c = self.code
        # A = P * F   (3x4 affine composition)
        A = [[None] * 4 for _ in range(3)]
        for i in range(3):
            for k in range(3):
                A[i][k] = c.tmp(c.dot([(P[i][m], F[m][k]) for m in range(3)]), f"a{j}_")
            A[i][3] = c.tmp(c.dot([(P[i][m], F[m][3]) for m in range(3)] + [(P[i][3], 1.0)]), f"a{j}_")
        q = f"q[{j}]"
        T = [[None] * 4 for _ in range(3)]
        if jt["type"] == "revolute":
            # T = A * Rz(q): columns 0 and 1 rotate, column 2 and the origin stay
            s, co = f"s{j}", f"c{j}"
            c.lines.append(f"float {s}, {co};")
            c.lines.append(f"sincosf({q}, &{s}, &{co});")
            for i in range(3):
                T[i][0] = c.tmp(c.dot([(co, A[i][0]), (s, A[i][1])]), f"t{j}_")
                T[i][1] = c.tmp(_sub(c, c.dot([(co, A[i][1])]), c.dot([(s, A[i][0])])), f"t{j}_")
                T[i][2] = A[i][2]
                T[i][3] = A[i][3]
        else:
            # T = A * Tz(q): the origin slides along column 2
            for i in range(3):
                T[i][0], T[i][1], T[i][2] = A[i][0], A[i][1], A[i][2]
                T[i][3] = c.tmp(c.dot([(A[i][3], 1.0), (q, A[i][2])]), f"t{j}_")
        self.frames[j] = T
        return T

    def point(self, f, xyz):
        """World coordinates of a point given in frame f."""
        T = self.frame(f)
        return [self.code.tmp(self.code.dot([(T[i][k], float(xyz[k])) for k in range(3)] + [(T[i][3], 1.0)]), "p")
                for i in range(3)]

    def relative(self, fa, fb):
        """Tab = inv(T_fa) * T_fb as a 3x4 of operands."""
        c = self.code
        Ta, Tb = self.frame(fa), self.frame(fb)
        d = [c.tmp(_sub(c, Tb[i][3], Ta[i][3]), "d") for i in range(3)]
        M = [[None] * 4 for _ in range(3)]
        for i in range(3):
            for k in range(3):
                M[i][k] = c.tmp(c.dot([(Ta[m][i], Tb[m][k]) for m in range(3)]), "r")
            M[i][3] = c.tmp(c.dot([(Ta[m][i], d[m]) for m in range(3)]), "r")
        return M


def _sub(c: _Code, a, b):
    """a - b over operands/expressions (strings are wrapped)."""
    if isinstance(a, float) and isinstance(b, float):
        return a - b
    if isinstance(b, float):
        if b == 0.0:
            return a
        return f"({a}) - {_lit(b)}" if b > 0 else f"({a}) + {_lit(-b)}"
    if isinstance(a, float) and a == 0.0:
        return f"-({b})"
    return f"({a}) - ({b})"


def _frame_arg(M):
    vals = []
    for i in range(3):
        for k in range(4):
            v = M[i][k]
            vals.append(_lit(v) if isinstance(v, float) else v)
    return "Frame{{" + ", ".join(vals) + "}}"


def emit_cuda_checker(m: dict) -> str:
    name = m["robot"]
    R = name.capitalize()
    sp = m["spheres"]
    code = _Code()
    fk = _FkGen(m, code)
    body = []

    # leaf tables: env leaves grouped into same-frame blocks; self pairs into
    # same-(frame a, frame b) blocks.  Blocks keep the reference's order.
    leaf_rows, pair_rows = [], []
    env_blocks, self_blocks = {}, {}
    for gi, g in enumerate(m["env_groups"]):
        blocks = []
        for leaf in g["leaves"]:
            f = sp[leaf]["frame"]
            if not blocks or blocks[-1][0] != f:
                blocks.append([f, len(leaf_rows), 0])
            s = sp[leaf]
            leaf_rows.append((s["c"][0], s["c"][1], s["c"][2], s["r"]))
            blocks[-1][2] += 1
        env_blocks[gi] = blocks
    for gi, g in enumerate(m["self_groups"]):
        blocks = []
        for a, b in g["pairs"]:
            fa, fb = sp[a]["frame"], sp[b]["frame"]
            if not blocks or (blocks[-1][0], blocks[-1][1]) != (fa, fb):
                blocks.append([fa, fb, len(pair_rows), 0])
            pair_rows.append((sp[a]["c"], sp[a]["r"], sp[b]["c"], sp[b]["r"]))
            blocks[-1][3] += 1
        self_blocks[gi] = blocks

    def env_block_calls(gi):
        """Leaf tests of an environment group: blocks of up to INLINE_LEAVES
        spheres are tested inline (centres folded at generation time), larger
        ones through ctx.env_leaves over the leaf table."""
        calls = []
        for f, first, n in env_blocks[gi]:
            T = fk.frame(f)
            if n <= INLINE_LEAVES:
                for k in range(first, first + n):
                    x, y, z, r = leaf_rows[k]
                    p = fk.point(f, (x, y, z))
                    calls.append(f"ctx.env_hit({_op(p[0])}, {_op(p[1])}, {_op(p[2])}, {_lit(r)})")
            else:
                calls.append(f"ctx.env_leaves({_frame_arg(T)}, k{R}Leaf + {first}, {n})")
        return calls

    table = name in TABLE_ROBOTS
    inline = not table or name in INLINE_VALIDATE
    # the gate spheres (environment groups' bounding spheres and self groups'
    # bounding pairs), each once, in order of first use
    gate_ids = {}
    for g in m["env_groups"]:
        if g["gate"] >= 0:
            gate_ids.setdefault(g["gate"], len(gate_ids))
    for g in m["self_groups"]:
        for sidx in g["gate"]:
            gate_ids.setdefault(sidx, len(gate_ids))
    # for the fast form the leaves of an ungated environment group stand in for its gate
    near_ids = dict(gate_ids)
    for g in m["env_groups"]:
        if g["gate"] < 0:
            for leaf in g["leaves"]:
                near_ids.setdefault(leaf, len(near_ids))
    tcode = None
    if table:
        # every frame, in chain order, into F[q + 1]; then the schedule loop
        nj = len(m["joints"])
        frames = [fk.frame(jt["q"]) for jt in m["joints"]]
        code.lines.append(f"FrameStore<Ctx, {nj + 1}> F(ctx);")
        code.lines.append("F.set(0, Frame{{1.0f, 0.0f, 0.0f, 0.0f, 0.0f, 1.0f, 0.0f, 0.0f, 0.0f, 0.0f, 1.0f, 0.0f}});")
        for jt, T in zip(m["joints"], frames):
            code.lines.append(f"F.set({jt['q'] + 1}, {_frame_arg(T)});")
        # gate centres in world coordinates, from the frames still in registers
        # (the schedule walk then reads 16 bytes per gate test, not a frame)
        fexpr = {-1: "world_frame()"} | {jt["q"]: _frame_arg(T) for jt, T in zip(m["joints"], frames)}
        code.lines.append(f"float4 G[{max(1, len(gate_ids))}];")
        for sidx, gid in gate_ids.items():
            code.lines.append(f"G[{gid}] = gate_centre({fexpr[sp[sidx]['frame']]}, k{R}Gate[{gid}]);")
        code.lines.append(f"return run_schedule(F.view(), G, schedule(marks, k{R}Sched, k{R}Step), {len(m['schedule'])}, k{R}EnvGroup, k{R}LeafBlock, k{R}Leaf, "
                          f"k{R}SelfGroup, k{R}PairBlock, k{R}Pair, ctx, marks);")
        tcode = code
        code = _Code()              # the straight-line form, if any, goes to its own code
        fk = _FkGen(m, code)
    for kind, gi in (m["schedule"] if inline else []):
        if kind == "env":
            g = m["env_groups"][gi]
            code.lines.append(f"// environment group {gi}: {g['label']}")
            for f, _, _ in env_blocks[gi]:       # frames are shared: compute outside the if
                fk.frame(f)
            if g["gate"] >= 0:
                s = sp[g["gate"]]
                x, y, z = fk.point(s["frame"], s["c"])
                code.lines.append(f"if (ctx.env_hit({_op(x)}, {_op(y)}, {_op(z)}, {_lit(s['r'])})) {{")
                for call in env_block_calls(gi):
                    code.lines.append(f"    if ({call}) return false;")
                code.lines.append("}")
            else:
                for call in env_block_calls(gi):
                    code.lines.append(f"if ({call}) return false;")
        else:
            g = m["self_groups"][gi]
            code.lines.append(f"// self group {gi}: {g['label']}")
            a, b = g["gate"]
            sa, sb = sp[a], sp[b]
            pa = fk.point(sa["frame"], sa["c"])
            pb = fk.point(sb["frame"], sb["c"])
            for fa, fb, _, _ in self_blocks[gi]:  # frames are shared: compute outside the if
                fk.frame(fa)
                fk.frame(fb)
            dx, dy, dz = (code.tmp(_sub(code, pa[i], pb[i]), "g") for i in range(3))
            code.lines.append(f"if (ctx.pair_hit({_op(dx)}, {_op(dy)}, {_op(dz)}, {_lit(sa['r'])} + {_lit(sb['r'])})) {{")
            for fa, fb, first, n in self_blocks[gi]:
                M = fk.relative(fa, fb)
                code.lines.append(f"    if (ctx.self_pairs({_frame_arg(M)}, k{R}Pair + {first}, {n})) return false;")
            code.lines.append("}")
        code.lines.append("if (ctx.stop()) return true;")
    if inline:
        code.lines.append("return true;")

    # fk_spheres: every sphere's world centre (not on the validation hot path)
    code2 = _Code()
    fk2 = _FkGen(m, code2)
    for i, s in enumerate(sp):
        x, y, z = fk2.point(s["frame"], s["c"])
        code2.lines.append(f"out[{i}] = make_float4({_op(x)}, {_op(y)}, {_op(z)}, {_lit(s['r'])});")

    out = []
    w = out.append
    w(f"// Straight-line CUDA collision checker for pRRTC's {name} model.  Generated by")
    w("// prrtc_gb300/robots/codegen.py from the fitted model; do not edit.")
    w("// Semantics follow the reference checker fkcc<Robot> (src/planning/utils.cuh):")
    w("// a leaf counts only when its group's gate (bounding sphere or bounding pair)")
    w("// is hit; a config is free when no counted leaf is hit.")
    w("#pragma once")
    if table:
        w('#include "../near_check.cuh"')
    w("")
    w(f"namespace prrtc {{ namespace gen_{name} {{")
    w("")
    w(f"constexpr int kDof = {m['dof']};")
    w(f"constexpr int kFrames = {len(m['joints']) + 1};   // the world and one frame per joint")
    w(f"constexpr int kNumSpheres = {len(sp)};")
    w(f"constexpr int kNumLeaves = {max(1, len(leaf_rows))};")
    w(f"constexpr int kNumPairs = {max(1, len(pair_rows))};")
    w("// canonical algorithmic FLOPs of one forward kinematics: 2 * (12 * dof + 9 * spheres)")
    w(f"constexpr unsigned kFkFlops = {2 * (12 * m['dof'] + 9 * len(sp))}u;")
    w("")
    w("// leaf spheres in their frame: (x, y, z, r)")
    w(f"__device__ const float4 k{R}Leaf[kNumLeaves] = {{")
    for r in leaf_rows or [(0.0, 0.0, 0.0, 0.0)]:
        w("    {%s}," % ", ".join(_lit(v) for v in r))
    w("};")
    w("// sphere pairs: a = (x, y, z, r) in frame A, b = (x, y, z, r) in frame B")
    w(f"__device__ const LeafPair k{R}Pair[kNumPairs] = {{")
    for ca, ra, cb, rb in pair_rows or [([0, 0, 0], 0.0, [0, 0, 0], 0.0)]:
        w("    {{%s, %s, %s, %s}, {%s, %s, %s, %s}}," % (*[_lit(v) for v in ca], _lit(ra), *[_lit(v) for v in cb], _lit(rb)))
    w("};")
    if table:
        w("// the schedule in table form (run_schedule)")
        w(f"__device__ const GenSched k{R}Sched[{len(m['schedule'])}] = {{")
        ne = ns = 0
        for kind, gi in m["schedule"]:
            n = _env_tests(m, gi) if kind == "env" else len(m["self_groups"][gi]["pairs"])
            ne, ns = (ne + n, ns) if kind == "env" else (ne, ns + 1)
            assert max(ne, ns) < 1 << 15, "GenSched's counts are 16 bits wide"
            w(f"    {{{{{0 if kind == 'env' else 1}, {gi}}}, {ne}, {ns}, {n}}},")
        w("};")
        w(f"__device__ const GenStep k{R}Step[{len(m['schedule'])}] = {{")
        for i in range(0, len(m["schedule"]), 8):
            w("    " + " ".join("{%d, %d}," % (0 if k == "env" else 1, g) for k, g in m["schedule"][i:i + 8]))
        w("};")
        lblocks, eg_rows = [], []
        for gi, g in enumerate(m["env_groups"]):
            first = len(lblocks)
            for f, fl, n in env_blocks[gi]:
                lblocks.append((f, fl, n))
            eg_rows.append((gate_ids[g["gate"]] if g["gate"] >= 0 else -1, first, len(lblocks) - first))
        w("// gate spheres (x, y, z, r) in their frames; gate_centre() puts them in the world")
        w(f"__device__ const float4 k{R}Gate[{max(1, len(gate_ids))}] = {{")
        for sidx in gate_ids or [None]:
            c = sp[sidx] if sidx is not None else {"c": [0.0, 0.0, 0.0], "r": 0.0}
            w("    {%s, %s, %s, %s}," % (*[_lit(v) for v in c["c"]], _lit(c["r"])))
        w("};")
        w(f"__device__ const GenEnvGroup k{R}EnvGroup[{max(1, len(eg_rows))}] = {{")
        for gid, first, nb in eg_rows or [(-1, 0, 0)]:
            w(f"    {{{gid}, {first}, {nb}, 0}},")
        w("};")
        w(f"__device__ const GenLeafBlock k{R}LeafBlock[{max(1, len(lblocks))}] = {{")
        for f, fl, n in lblocks or [(-1, 0, 0)]:
            w(f"    {{{f}, {fl}, {n}, 0}},")
        w("};")
        pblocks, sg_rows = [], []
        for gi, g in enumerate(m["self_groups"]):
            first = len(pblocks)
            for fa, fb, pf, n in self_blocks[gi]:
                pblocks.append((fa, fb, pf, n))
            a, b = g["gate"]
            sg_rows.append((gate_ids[a], gate_ids[b], first, len(pblocks) - first))
        w(f"__device__ const GenSelfGroup k{R}SelfGroup[{max(1, len(sg_rows))}] = {{")
        for ga, gb, first, nb in sg_rows or [(0, 0, 0, 0)]:
            w(f"    {{{ga}, {gb}, {first}, {nb}}},")
        w("};")
        w(f"__device__ const GenPairBlock k{R}PairBlock[{max(1, len(pblocks))}] = {{")
        for fa, fb, pf, n in pblocks or [(-1, -1, 0, 0)]:
            w(f"    {{{fa}, {fb}, {pf}, {n}}},")
        w("};")
        w("// the same for the fast form (near_check.cuh)")
        w(f"__device__ const NearPairBlock k{R}NearPair[{max(1, len(pblocks))}] = {{")
        for fa, fb, pf, n in pblocks or [(-1, -1, 0, 0)]:
            row, c, r = _rows(pair_rows[pf:pf + n])
            w(f"    {{{fa}, {fb}, {pf}, {n}, {{{', '.join(_lit(v) for v in [*c, r])}}}, {row}}},")
        w("};")
    w("")

    def function(head, lines, more="", types="class Ctx"):
        w(f"template <{types}>")
        w(f"{head}(const float *__restrict__ q, Ctx &ctx{more})")
        w("{")
        for line in lines:
            w("    " + line)
        w("}")
        w("")

    def fast_or(exact):
        """The fast form's answer, else the exact form's (on values the
        compiler cannot tell from new ones, so that it keeps none of the fast
        form's kinematics for them)."""
        call = [f"if constexpr (Ctx::kInlineExact) return {exact}(c, ctx, marks);",
                "Ctx own = ctx;   // the call must not force the caller's into memory",
                f"const bool free = {exact}_call(c, own, marks);", "ctx.work = own.work;", "return free;"]
        if exact != "fkcc_exact":   # single configurations: always compiled into the kernel
            call = [f"return {exact}(c, ctx, marks);"]
        return [f"if constexpr (Ctx::kEveryTest) return {exact}(q, ctx, AllSteps{{}});",
                f"StepMarks<{(len(m['schedule']) + 31) // 32}> marks;   // the steps that the exact form has to make",
                "const int a = near_check(q, ctx, marks);", "if (a != kNearUnsure) return a == kNearFree;", "float c[kDof];",
                "#pragma unroll", "for (int d = 0; d < kDof; d++) {", "    c[d] = q[d];",
                '    asm volatile("" : "+f"(c[d]));', "}", *call]

    if table:
        near_gates = near_ids
        marks_type = f"StepMarks<{(len(m['schedule']) + 31) // 32}>"
        w(f"struct {R}Near {{")
        w(f"    static constexpr int kDof = {m['dof']}, kFrames = {len(m['joints'])}, kGates = {len(near_gates)}, "
          f"kWords = {(len(m['schedule']) + 31) // 32};")
        for name_, type_, arr in (("steps", "GenSched", "Sched"), ("env_groups", "GenEnvGroup", "EnvGroup"),
                                  ("leaf_blocks", "GenLeafBlock", "LeafBlock"), ("leaves", "float4", "Leaf"),
                                  ("self_groups", "GenSelfGroup", "SelfGroup"), ("pair_blocks", "NearPairBlock", "NearPair"),
                                  ("pairs", "LeafPair", "Pair")):
            w(f"    static __device__ __forceinline__ const {type_} *{name_}() {{ return k{R}{arr}; }}")
        w("    static __device__ __forceinline__ void frames(const float *q, NearFrame *F, float4 *G)")
        w("    {")
        for line in _near_frames(m, near_gates):
            w("        " + line)
        w("    }")
        w("};")
        w("")
        w("// The exact form; marks: the steps to make (StepMarks), or AllSteps.")
        function("__device__ __forceinline__ bool fkcc_exact", tcode.lines, ", const Marks &marks", "class Ctx, class Marks")
        function("__device__ __noinline__ bool fkcc_exact_call", ["return fkcc_exact(q, ctx, marks);"], f", const {marks_type} marks")
        if inline:
            w("// The straight-line exact form makes every step, whatever the marks.")
            function("__device__ __forceinline__ bool fkcc_validate_exact", code.lines, ", const Marks &", "class Ctx, class Marks")
        out_marks = f", {marks_type} &marks"
        function("__device__ __forceinline__ int near_check_leaves", _near_body(m, near_gates, LEAF_MARKS), out_marks)
        function("__device__ __forceinline__ int near_check_gates", _near_body(m, near_gates, ALWAYS), out_marks)
        function("__device__ __forceinline__ int near_check",
                 ["if constexpr (Ctx::kLeafMarks) return near_check_leaves(q, ctx, marks);",
                  "else return near_check_gates(q, ctx, marks);"], out_marks)
    w("// Returns true when configuration q is collision-free.")
    function("__device__ __forceinline__ bool fkcc", fast_or("fkcc_exact") if table else code.lines)
    w("// The same verdicts for the stand-alone checker of single configurations.")
    function("__device__ __forceinline__ bool fkcc_validate",
             fast_or("fkcc_validate_exact") if table and inline else ["return fkcc(q, ctx);"])
    w("// Row i (0..2) of every joint's world frame in pairs of floats, joint at table")
    w("// position j at hi / lo[12 j + 4 i + k]; trig: cosine and sine of each joint's")
    w("// angle, or its value (clearance_eval.cuh).")
    w("template <class Dd>")
    w("__device__ __forceinline__ void clr_rows(int i, const Dd *__restrict__ trig, float *__restrict__ hi, float *__restrict__ lo)")
    w("{")
    for line in _clr_rows(m):
        w("    " + line)
    w("}")
    w("")
    w("// World centre and radius of every model sphere (model sphere order).")
    w("__device__ __forceinline__ void fk_spheres(const float *__restrict__ q, float4 *__restrict__ out)")
    w("{")
    for line in code2.lines:
        w("    " + line)
    w("}")
    w("")
    w(f"}} }}  // namespace prrtc::gen_{name}")
    w("")
    return "\n".join(out)


def _bounding_sphere(spheres):
    """(centre, radius) of a sphere around the given (centre, radius) spheres,
    the radius rounded up."""
    c = np.mean([s[0] for s in spheres], axis=0)
    for k in range(2000):          # towards the farthest one, by shrinking steps
        d = [round(float(np.linalg.norm(np.asarray(x) - c)) + r, 9) for x, r in spheres]
        i = int(np.argmax(d))
        v = np.asarray(spheres[i][0]) - c
        n = np.linalg.norm(v)
        if n < 1e-9:
            break
        c = c + v / n * min(n, d[i] * 0.5 / (k + 2))
    c = np.round(c, 4)
    r = max(float(np.linalg.norm(np.asarray(x) - c)) + r for x, r in spheres)
    return [float(x) for x in c], float(np.ceil(r * 1e5 + 1.0) / 1e5)


GRID_UNIT = 512        # kGridUnit, device_common.cuh
NEAR_PAD = 1e-4        # kNearPad, near_check.cuh
LEAF_MARKS = 0.03      # gate pairs that overlap in this share of random configurations get leaf marks
ALWAYS = 0.9           # and above this the gates are not asked first
WIDE = 0.19            # spheres above EnvGrid::out_r (env_grid.cu: 0.95 x 0.2 m)
CLUSTER = 3            # gate pairs of two frames that are worth a test of the frames' gates as a whole


def _near_frames(m, gate_ids):
    """Every frame and gate centre into the walk's arrays (near_resolve)."""
    code = _Code()
    fk = _FkGen(m, code)
    sp, w = m["spheres"], code.lines.append
    frames = {-1: "world_frame()"}
    for jt in m["joints"]:
        frames[jt["q"]] = _frame_arg(fk.frame(jt["q"]))
        w(f"F[{jt['q']}].set({frames[jt['q']]});")
    for sidx, gid in gate_ids.items():
        w(f"G[{gid}] = gate_centre({frames[sp[sidx]['frame']]}, {_sphere_arg(sp[sidx])});")
    return [line.replace("sincosf(", "near_sincos(") for line in code.lines]


def _sphere_arg(s):
    return f"make_float4({', '.join(_lit(float(np.float32(v))) for v in (*s['c'], s['r']))})"


def _near_body(m, gate_ids, leaf_marks):
    """The fast form (near_check.cuh): frames, gate centres and the marks of the
    schedule's steps that can hit, in chain order; then the walk, for lanes
    with marked steps.  Self groups whose gates overlap in at least this share
    of random configurations get leaf marks."""
    R = m["robot"].capitalize()
    code = _Code()
    fk = _FkGen(m, code)
    sp, w = m["spheres"], code.lines.append
    steps = m["schedule"]
    words = (len(steps) + 31) // 32
    w("const EnvGrid *grid = ctx.env.grid;")
    w("#pragma unroll")
    w(f"for (int w = 0; w < {words}; w++) marks.marked[w] = ~0u, marks.passed[w] = 0u;")
    w("if (!grid || !(grid->lo[0] <= grid->hi[0])) return kNearUnsure;")
    w(f"if (!({' + '.join(f'fabsf(q[{d}])' for d in range(m['dof']))} < 100.0f)) return kNearUnsure;")
    for jt in m["joints"]:
        if jt["type"] != "revolute":
            w(f"if (fabsf(q[{jt['q']}]) > 4.0f) return kNearUnsure;")
    w("const NearView near = near_view(ctx);")
    w("unsigned " + ", ".join(f"m{k} = 0, p{k} = 0" for k in range(words)) + ";   // marked and passed steps")
    w("int extra = 0;   // FLOPs of the passed steps' leaf pairs")

    def mark(s, cond):
        return f"m{s >> 5} |= {cond} ? {hex(1 << (s & 31))}u : 0u;"

    env_of = {}     # sphere -> environment steps that it gates
    for s, (kind, gi) in enumerate(steps):
        if kind == "env":
            g = m["env_groups"][gi]
            for sidx in ([g["gate"]] if g["gate"] >= 0 else g["leaves"]):
                env_of.setdefault(sidx, []).append(s)
    fexpr = {-1: "world_frame()"}
    for f in [-1] + [jt["q"] for jt in m["joints"]]:
        if f >= 0:
            fexpr[f] = _frame_arg(fk.frame(f))
        for sidx, gid in gate_ids.items():
            if sp[sidx]["frame"] != f:
                continue
            w(f"const float4 g{gid} = gate_centre({fexpr[f]}, {_sphere_arg(sp[sidx])});")
            r = np.float32(sp[sidx]["r"])
            for s in env_of.get(sidx, []):
                w(mark(s, f"may_hit_env{'_wide' if r >= WIDE else ''}(near, g{gid}, {int(np.ceil(float(r) * GRID_UNIT))})"))

    pairs = {}
    for s, (kind, gi) in enumerate(steps):
        if kind != "env":
            a, b = m["self_groups"][gi]["gate"]
            key = tuple(sp[x]["frame"] if sp[x]["frame"] >= 0 else ("world", x) for x in (a, b))
            pairs.setdefault(key, []).append((s, a, b))
    clusters = {}

    def cluster(key, gates):
        """The centre of the sphere around a frame's gates, emitted once."""
        if not isinstance(key, int) or len(gates) == 1:
            return f"g{gate_ids[gates[0]]}"
        name = f"b{key}_" + "_".join(str(gate_ids[x]) for x in gates)
        if name not in clusters:
            c, r = _bounding_sphere([(np.float32(sp[x]["c"]).astype(float), float(np.float32(sp[x]["r"]))) for x in gates])
            clusters[name] = f"c{key}_{len(clusters)}"
            w(f"const float4 {clusters[name]} = gate_centre({fexpr[key]}, make_float4({', '.join(_lit(v) for v in [*c, r])}));")
        return clusters[name]

    often = _gate_rates(m)

    def test(s, a, b):
        """The mark of self step s (gates a, b): by its gates, or, where those
        overlap often, by its leaves."""
        gi = steps[s][1]
        gates = f"may_hit_pair(near, g{gate_ids[a]}, g{gate_ids[b]})"
        if often[gi] < leaf_marks:
            return [mark(s, gates)]
        lines = []
        for frame, balls in _leaf_marks(m, gi):
            for (f, c, r), limits in balls:
                ball = f"gate_centre({fexpr[f]}, make_float4({', '.join(_lit(v) for v in [*c, r])}))"
                lines.append(f"{{ const float4 p = local_point({fexpr[frame]}, {ball});")
                lines += [f"  n |= near_leaf(p, {', '.join(_lit(v) for v in row)});" for row in limits]
                lines.append("}")
        bit, k = f"{hex(1 << (s & 31))}u", s >> 5
        body = ["    bool n = near.wide || h == 2;", *("    " + x for x in lines), f"    if (n) m{k} |= {bit};",
                f"    else if (h) p{k} |= {bit}, extra += kFlopPair * {len(m['self_groups'][gi]['pairs'])};", "}"]
        head = f"const int h = near_gate(near, g{gate_ids[a]}, g{gate_ids[b]});"
        if often[gi] > ALWAYS:
            return [f"{{   {head}", *body]
        return [f"if ({head[:-1]}) {{", *body]

    for (ka, kb), list_ in pairs.items():
        tests = [x for s, a, b in list_ for x in test(s, a, b)]
        if len(list_) >= CLUSTER:
            ca = cluster(ka, sorted({a for _, a, _ in list_}))
            cb = cluster(kb, sorted({b for _, _, b in list_}))
            w(f"if (may_hit_pair(near, {ca}, {cb})) {{")
            code.lines += ["    " + t for t in tests]
            w("}")
        else:
            code.lines += tests
    any_ = " | ".join(f"m{k}" for k in range(words))
    env_total = sum(_env_tests(m, gi) for kind, gi in steps if kind == "env")
    self_total = sum(kind != "env" for kind, _ in steps)
    for k in range(words):
        w(f"marks.marked[{k}] = m{k}, marks.passed[{k}] = p{k};")
    w(f"if ({any_}) {{")
    w("    if (ctx.stop()) return kNearFree;")
    w(f"    const unsigned a = near_resolve<{R}Near>(NearCfg<kDof>{{{{{', '.join(f'q[{d}]' for d in range(m['dof']))}}}}}, marks, extra, grid, ctx.pad);")
    w("    if ((a & 3u) == kNearHit) ctx.work += a >> 2;")
    w("    if ((a & 3u) != kNearFree) return (int)(a & 3u);")
    w("    extra = (int)a >> 2;")
    w("}")
    w(f"ctx.work += (unsigned)(grid->cost * {env_total} + kFlopPair * {self_total} + extra);")
    w("return kNearFree;")
    return [line.replace("sincosf(", "near_sincos(") for line in code.lines]


def _gate_rates(m):
    """Share of random configurations in which each self group's gates overlap."""
    from .. import scenes
    q = scenes._uniform_configs(m["robot"], scenes.Rng(1), 2048)
    C = scenes.sphere_centres(m["robot"], q)
    r = [s["r"] for s in m["spheres"]]
    return [float((((C[a] - C[b]) ** 2).sum(-1) < (r[a] + r[b]) ** 2).mean()) for a, b in (g["gate"] for g in m["self_groups"])]


def _balls(spheres):
    """A few balls [(centre, radius)] around (centre, radius) spheres, tighter
    than one: grouped by the nearest of seeds that are far from one another."""
    P = np.array([c for c, _ in spheres])
    k = min(len(P), 3) if len(P) > 2 else 1
    seeds = [int(np.argmax(((P - P.mean(0)) ** 2).sum(1)))]
    while len(seeds) < k:
        seeds.append(int(np.argmax(np.min([((P - P[i]) ** 2).sum(1) for i in seeds], axis=0))))
    cen = P[seeds]
    for _ in range(8):
        of = np.argmin(((P[:, None] - cen) ** 2).sum(-1).round(9), 1)
        cen = np.array([P[of == i].mean(0) if (of == i).any() else cen[i] for i in range(k)])
    return [_bounding_sphere([spheres[j] for j in range(len(P)) if of[j] == i]) for i in range(k) if (of == i).any()]


def _leaf_marks(m, gi):
    """Leaf tests of a self group: [(frame, [((ball's frame, centre, radius),
    [(-2 a, limit) per leaf a of `frame`])])], see near_check.cuh."""
    sp = m["spheres"]
    f32 = lambda v: float(np.float32(v))  # noqa: E731
    sph = lambda i: ([f32(x) for x in sp[i]["c"]], f32(sp[i]["r"]))  # noqa: E731
    A, B = (sorted({p[k] for p in m["self_groups"][gi]["pairs"]}) for k in (0, 1))
    if len(A) > len(B):
        A, B = B, A      # the longer list is enclosed in balls
    balls = []
    for f in sorted({sp[i]["frame"] for i in B}):
        balls += [(f, c, r) for c, r in _balls([sph(i) for i in B if sp[i]["frame"] == f])]
    out = []
    for f in sorted({sp[i]["frame"] for i in A}):
        tests = []
        for ball in balls:
            rows = []
            for i in (i for i in A if sp[i]["frame"] == f):
                a, r = sph(i)
                s = r + ball[2] + 2 * NEAR_PAD + 2e-5
                rows.append([-2 * x for x in a] + [round(s * s - sum(x * x for x in a) + 2e-6, 7)])
            tests.append((ball, rows))
        out.append((f, tests))
    return out


def _rows(rows):
    """(row, centre, radius) of a block of pairs (ca, ra, cb, rb): `row` pairs
    per sphere a, every a against the same spheres b, which the sphere
    (centre, radius) encloses; row = 0 where the block is not of that form or
    skipping rows saves nothing."""
    f = lambda v: [float(np.float32(x)) for x in v]  # noqa: E731
    a = [(tuple(r[0]), r[1]) for r in rows]
    b = [(tuple(r[2]), r[3]) for r in rows]
    row = next((k for k in range(1, len(a)) if a[k] != a[0]), len(a))
    if row < 3 or len(a) % row or len(a) // row > 32 or any(
            a[k] != a[k - k % row] or b[k] != b[k % row] for k in range(len(a))):
        return 0, [0.0, 0.0, 0.0], 0.0
    return row, *_bounding_sphere([(np.array(f(x)), float(np.float32(y))) for x, y in b[:row]])


def _clr_rows(m):
    """One row of every frame, fixed transforms folded (T = parent F Rz(q))."""
    f32 = lambda v: float(np.float32(v))  # noqa: E731
    out, w, rows = [], None, {}
    w = out.append
    for pos, jt in enumerate(m["joints"]):
        F = [[f32(v) for v in r] for r in jt["F"]]
        A = []
        for k in range(4):
            if jt["parent"] < 0:       # the world's row i is a unit vector
                c = [F[r][k] for r in range(3)]
                e = _lit(c[0]) if c[0] == c[1] == c[2] else f"i == 0 ? {_lit(c[0])} : i == 1 ? {_lit(c[1])} : {_lit(c[2])}"
                w(f"const Dd a{pos}_{k}{{{e}, 0.0f}};")
            else:
                P = rows[jt["parent"]]
                terms = [P[r] if F[r][k] == 1.0 else f"(-{P[r]})" if F[r][k] == -1.0 else f"{P[r]} * {_lit(F[r][k])}"
                         for r in range(3) if F[r][k] != 0.0] + ([P[3]] if k == 3 else [])
                w(f"const Dd a{pos}_{k} = {' + '.join(terms) if terms else 'Dd{0.0f, 0.0f}'};")
            A.append(f"a{pos}_{k}")
        if jt["type"] == "revolute":
            w(f"const Dd c{pos} = trig[{2 * pos}], s{pos} = trig[{2 * pos + 1}];")
            w(f"const Dd t{pos}_0 = c{pos} * {A[0]} + s{pos} * {A[1]}, t{pos}_1 = c{pos} * {A[1]} - s{pos} * {A[0]};")
            T = [f"t{pos}_0", f"t{pos}_1", A[2], A[3]]
        else:
            w(f"const Dd t{pos}_3 = {A[3]} + {A[2]} * trig[{2 * pos}].h;")
            T = [A[0], A[1], A[2], f"t{pos}_3"]
        rows[jt["q"]] = T
        for k in range(4):
            w(f"hi[{12 * pos + k} + 4 * i] = {T[k]}.h, lo[{12 * pos + k} + 4 * i] = {T[k]}.l;")
    return out


def _env_tests(m, gi):
    """Spheres of an environment group tested when nothing hits."""
    g = m["env_groups"][gi]
    return 1 if g["gate"] >= 0 else len(g["leaves"])


def _op(v):
    return _lit(v) if isinstance(v, float) else v


def write_all():
    for r in ROBOTS:
        m = load_model(r)
        (CSRC / f"{r}_model.h").write_text(emit_c_tables(m))
        (CSRC / f"{r}_fkcc.cuh").write_text(emit_cuda_checker(m))


def check_up_to_date() -> list:
    """Names of generated files that differ from what the JSON models give."""
    stale = []
    for r in ROBOTS:
        m = load_model(r)
        for path, text in ((CSRC / f"{r}_model.h", emit_c_tables(m)), (CSRC / f"{r}_fkcc.cuh", emit_cuda_checker(m))):
            if not path.exists() or path.read_text() != text:
                stale.append(path.name)
    return stale


if __name__ == "__main__":
    write_all()
