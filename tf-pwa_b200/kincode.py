"""Kinematics compiler: emits the CUDA source of a model's dataset step.

Two device functions are generated per model, straight-line code in FP64:

``model_kin(P, F)``     final-state four-momenta (parent rest frame, in
                        ``dat_order``) -> every event field of the plan:
                        invariant masses, helicity angles per decay and
                        alignment angles of spinning finals.  It is the
                        algorithm of ``kinematics.event_fields`` (which
                        restates ``tf_pwa/cal_angle.py:158-251,262-343,
                        346-378,408-490``), unrolled over the model's
                        topologies: node momenta, successive rest-frame
                        momenta, Euler angles with the alpha range bias per
                        out, SU(2) rotation/boost products for alignment.
``model_genbod(U, P)``  one flat phase-space event from uniforms U by the
                        Raubold-Lynch (GENBOD) construction of
                        ``phasespace.generate_weighted`` (the role of
                        ``tf_pwa/phasespace.py:31-368``, with its chain
                        generator for fixed-mass intermediates); returns
                        the event weight over its upper bound.

Generation levels: the parent, and every fixed-mass intermediate that the
reference's phase-space sampler also generates on shell (a node common to
all topologies whose particle has model "one"), each decayed in its own rest
frame and boosted.  Uniform draws of an event, level by level (depth first):
k - 2 sorted uniforms for the intermediate masses of a k-body level, then
(cos theta, phi) of each of its k - 1 splittings; then the phase-space
accept draw (against the product of the levels' weights over their upper
bounds) and the amplitude accept draw.
"""
import math

from .plan import split_swap


def _f(v):
    r = repr(float(v))
    if "e" not in r and "." not in r and "inf" not in r and "nan" not in r:
        r += ".0"
    return r


def _pdk(a, b, c):
    x = (a - b - c) * (a + b + c) * (a - b + c) * (a + b - c)
    return math.sqrt(max(x, 0.0)) / (2 * a)


class KinCode:
    def __init__(self, plan, order):
        self.plan = plan
        self.order = [str(o) for o in order]
        group = plan.group
        finals = {str(o): o for o in group.outs}
        missing = [o for o in self.order if o not in finals]
        if missing or len(self.order) != len(finals):
            raise ValueError(f"dat_order {self.order} does not list the final particles "
                             f"{sorted(finals)}")
        self.parent_mass = group.top.mass
        self.masses = [finals[o].mass for o in self.order]
        self.ok = self.parent_mass is not None and all(m is not None for m in self.masses)
        self.nfin = len(self.order)
        self.nfield = plan.n_fields
        self.levels = self._build_levels() if self.ok else [(self.parent_mass, [])]
        # per level of k bodies: k - 2 sorted uniforms + (cos theta, phi) per
        # splitting; then the phase-space and amplitude accept draws
        self.ndraw = sum(3 * len(b) - 4 for _, b in self.levels) + 2

    # ------------------------------------------------------------ kinematics
    def _wanted(self, sk):
        """What the fields of pass ``sk`` read: helicity angles as
        {(topology, decay, particle): [(field, "alpha" | "beta")]}, masses as
        {node name: field}, and the finals whose SU(2) path is needed as
        {(topology, final)} (alignment fields and their reference)."""
        plan = self.plan
        angles, masses, su2 = {}, {}, set()
        for fi, full_name in enumerate(plan.fields):
            if fi == plan.charge_index:
                continue
            k, fname = split_swap(full_name)
            parts = fname.split("/")
            if k != sk:
                continue
            if parts[0] == "m":
                masses[parts[1]] = fi
                continue
            t = int(parts[0])
            topo = plan.topos[t]
            dec = next(d for d in topo.chain if topo.decay_name(d) == parts[1])
            part = next(o for o in dec.outs if topo.node[o] == parts[2])
            if parts[3] == "aligned":
                su2.add((t, part))
                ref = plan.align_ref[str(part)]
                su2.add((ref, next(o for o in plan.topos[ref].chain.outs
                                   if str(o) == str(part))))
            else:
                angles.setdefault((t, dec, part), []).append((fi, parts[3]))
        return angles, masses, su2

    def _emit_pass(self, e, pexpr, sk):
        """Masses and helicity angles of one set of momenta (``pexpr``:
        final -> LV expression), each field written as soon as it is formed;
        what several topologies share (the parent's frame, finals in it) is
        emitted once.  Returns per topology the names of the finals' SU(2)
        rotation and boost products."""
        plan = self.plan
        want, masses, su2 = self._wanted(sk)
        n = [0]

        def tmp(prefix):
            n[0] += 1
            return f"p{sk}{prefix}{n[0]}"

        def lsum(parts):
            expr = parts[0]
            for p in parts[1:]:
                expr = f"lv_add({expr}, {p})"
            return expr

        for topo in plan.topos:
            for p in topo.chain.inner:
                fi = masses.pop(topo.node[p], None)
                if fi is not None:
                    fs = [pexpr[str(f)] for f in topo.chain.final_set(p)]
                    e(f"  F[{fi}] = kin_inv_mass({lsum(fs)});")
        outs = [str(o) for o in plan.topos[0].chain.outs]
        top, frame, axes = tmp("top"), tmp("fr"), tmp("ax")
        e(f"  const LV {top} = {lsum([pexpr[o] for o in outs])};")
        e(f"  const KBoost {frame} = kin_frame({top});")
        e(f"  const KAxes {axes} = kin_top_axes({top}, {'true' if plan.random_z else 'false'});")
        in_top = {}
        for o in outs:
            in_top[o] = tmp("q")
            e(f"  const LV {in_top[o]} = kin_to_rest({frame}, {pexpr[o]});")
        result = []
        for t, topo in enumerate(plan.topos):
            chain = topo.chain
            decay_of = {d.core: d for d in chain}
            path = {}  # particles on the way to a final whose SU(2) product is needed
            for tt, o in su2:
                if tt == t:
                    p = o
                    while p != chain.top:
                        path[p] = True
                        p = next(d for d in chain if p in d.outs).core
            rmat, bmat = {}, {}

            def need(d):
                """Whether the momenta of decay d's daughters are read."""
                return any((t, d, j) in want or j in path or (j in decay_of and need(decay_of[j]))
                           for j in d.outs)

            def walk(d, vec, ax, bm, rm):
                """Decay d with the finals' momenta ``vec`` in its mother's
                rest frame, the mother's axes and SU(2) products."""
                for i, j in enumerate(d.outs):
                    inner = j in decay_of and need(decay_of[j])
                    if not ((t, d, j) in want or j in path or inner):
                        continue
                    if j in decay_of:
                        v = tmp("n")
                        e(f"  const LV {v} = {lsum([vec[str(f)] for f in chain.final_set(j)])};")
                    else:
                        v = vec[str(j)]
                    a, x = tmp("a"), tmp("x")
                    e(f"  const KAngles {x} = kin_angles({ax}, lv_vec({v}));")
                    e(f"  const double {a} = kin_fold_{'first' if i == 0 else 'second'}"
                      f"({x}.alpha);")
                    b, x = f"{x}.beta", f"{x}.axes"
                    for fi, kind in want.get((t, d, j), ()):
                        e(f"  F[{fi}] = {a if kind == 'alpha' else b};")
                    nb = nr = None
                    if j in path:
                        nb, nr = tmp("B"), tmp("R")
                        e(f"  const SU2 {nb} = su2_boost_z_from_p({v});")
                        e(f"  const SU2 {nr} = " + (
                            f"su2_mul(su2_rot_yz({b}, {a}), su2_mul({bm}, {rm}));" if bm
                            else f"su2_rot_yz({b}, {a});"))
                        rmat[j], bmat[j] = nr, nb
                    if inner:
                        fr = tmp("fr")
                        e(f"  const KBoost {fr} = kin_frame({v});")
                        dj = decay_of[j]
                        sub = {}
                        for q in dj.outs:
                            if not ((t, dj, q) in want or q in path
                                    or (q in decay_of and need(decay_of[q]))):
                                continue
                            for f in (chain.final_set(q) if q in decay_of else [q]):
                                sub[str(f)] = tmp("r")
                                e(f"  const LV {sub[str(f)]} = kin_to_rest({fr}, {vec[str(f)]});")
                        walk(dj, sub, x, nb, nr)

            walk(decay_of[chain.top], in_top, axes, None, None)
            result.append((rmat, bmat))
        return result

    def _emit_kin(self, e):
        plan = self.plan
        fin = {o: i for i, o in enumerate(self.order)}
        # unswapped momenta, then one relabelling per swap (final pi takes the
        # momentum of src[pi], three-momentum reversed in the CP-conjugate ones)
        all_frames = [self._emit_pass(e, {o: f"P[{fin[o]}]" for o in fin}, 0)]
        for k, sw in enumerate(plan.swaps):
            pe = {}
            for o in fin:
                q = f"P[{fin[sw['src'].get(o, o)]}]"
                pe[o] = f"LV{{{q}.t, -{q}.x, -{q}.y, -{q}.z}}" if sw["neg"] else q
            all_frames.append(self._emit_pass(e, pe, k + 1))
        cnt = [0]
        aligned = {}  # Euler angle names of the alignment rotations emitted so far

        def tmp(prefix):
            cnt[0] += 1
            return f"{prefix}{cnt[0]}"

        # alignment angles, and the charge
        for fi, full_name in enumerate(plan.fields):
            if fi == plan.charge_index:
                # the event's charge is data, not kinematics: +1 here (the
                # generator's events), overwritten by the caller's charges
                e(f"  F[{fi}] = 1.0;")
                continue
            sk, fname = split_swap(full_name)
            parts = fname.split("/")
            if parts[-2] != "aligned":
                continue  # written with its decay
            tidx = int(parts[0])
            topo = plan.topos[tidx]
            dec = [d for d in topo.chain if topo.decay_name(d) == parts[1]][0]
            part = [o for o in dec.outs if topo.node[o] == parts[2]][0]
            rmat, bmat = all_frames[sk][tidx]
            ref_t = plan.align_ref[str(part)]
            rr, rb = all_frames[sk][ref_t]
            rpart = [o for o in plan.topos[ref_t].chain.outs if str(o) == str(part)][0]
            if (sk, tidx, part) not in aligned:
                m, al, be, ga = tmp("al_M"), tmp("al_a"), tmp("al_b"), tmp("al_g")
                e(f"  const SU2 {m} = su2_mul(su2_mul({rb[rpart]}, su2_mul({rr[rpart]}, "
                  f"su2_inv({rmat[part]}))), su2_inv({bmat[part]}));")
                e(f"  double {al}, {be}, {ga};")
                e(f"  su2_euler({m}, &{al}, &{be}, &{ga});")
                aligned[(sk, tidx, part)] = (al, be, ga)
            al, be, ga = aligned[(sk, tidx, part)]
            e(f"  F[{fi}] = {dict(alpha=al, beta=be, gamma=ga)[parts[4]]};")

    # ------------------------------------------------------------ GENBOD
    def _build_levels(self):
        """Generation structure.  As the reference's phase-space sampler
        (``tf_pwa/config_loader/sample.py:276-340``, build_phsp_chain), an
        inner node present in every topology whose particle has the fixed
        lineshape (model "one") and a mass is generated on shell: its
        daughters come from a two-(or more)-body decay in its rest frame.
        Levels in depth-first order, level 0 = the parent; each level is
        (mass, [(kind, ref, mass)]) with kind "f" (ref = index in dat_order)
        or "n" (ref = level index)."""
        plan = self.plan
        fin = {o: i for i, o in enumerate(self.order)}
        sets = None
        node_particle = {}
        for topo in plan.topos:
            here = set()
            for p in topo.chain.inner:
                fs = frozenset(str(f) for f in topo.chain.final_set(p))
                here.add(fs)
                node_particle.setdefault(fs, []).append(p)
            sets = here if sets is None else sets & here
        fixed = {}
        for fs in sets or ():
            ps = node_particle[fs]
            if all(p.lineshape_kind() == "one" and getattr(p, "model", None) == "one"
                   and p.mass is not None for p in ps):
                fixed[fs] = ps[0].mass
        levels = []

        def build(mass, finals):
            lid = len(levels)
            levels.append(None)
            inner = [fs for fs in fixed if fs < finals]
            # maximal fixed nodes inside this level
            tops = [fs for fs in inner if not any(fs < g for g in inner)]
            covered = set().union(*tops) if tops else set()
            bodies = [("f", fin[f], self.masses[fin[f]]) for f in finals - covered]
            for fs in tops:
                bodies.append(("n", fs, fixed[fs]))
            bodies.sort(key=lambda b: b[1] if b[0] == "f" else min(fin[f] for f in b[1]))
            out = []
            for kind, ref, m in bodies:
                if kind == "n":
                    ref = build(m, ref)
                out.append((kind, ref, m))
            levels[lid] = (mass, out)
            return lid

        build(self.parent_mass, frozenset(self.order))
        return levels

    def _emit_genbod(self, e):
        levels = self.levels
        draw = 0
        e("  double w = 1.0;")
        two_pi = _f(2 * math.pi)
        for lid, (M, bodies) in enumerate(levels):
            ms = [m for _, _, m in bodies]
            k = len(ms)
            tm = M - sum(ms)
            if tm <= 0:
                raise ValueError("a generation level is below the sum of its daughter masses")
            cum = [sum(ms[:i + 1]) for i in range(k)]
            emmax, emmin, wtmax = tm + ms[0], 0.0, 1.0
            for i in range(1, k):
                emmin += ms[i - 1]
                emmax += ms[i]
                wtmax *= _pdk(emmax, emmin, ms[i])
            pre = f"g{lid}_"
            e(f"  LV {pre}b[{k}];")
            e("  {")
            k2 = k - 2
            if k2 > 0:
                e(f"    double r[{k2}];")
                for j in range(k2):
                    e(f"    r[{j}] = U[{draw + j}];")
                for i in range(k2):
                    for j in range(k2 - 1 - i):
                        e(f"    {{ const double lo = fmin(r[{j}], r[{j + 1}]), hi = fmax(r[{j}], "
                          f"r[{j + 1}]); r[{j}] = lo; r[{j + 1}] = hi; }}")
            draw += k2
            e(f"    const double Ms0 = {_f(ms[0])};")
            for i in range(1, k - 1):
                e(f"    const double Ms{i} = r[{i - 1}] * {_f(tm)} + {_f(cum[i])};")
            e(f"    const double Ms{k - 1} = {_f(M)};")
            e("    double wl = 1.0;")
            for i in range(1, k):
                e(f"    const double pd{i} = kin_pdk(Ms{i}, Ms{i - 1}, {_f(ms[i])});")
                e(f"    wl *= pd{i};")
            for i in range(1, k):
                cu, pu = draw, draw + 1
                draw += 2
                e(f"    {{ const double cth = 2.0 * U[{cu}] - 1.0, phi = {two_pi} * U[{pu}];")
                e("      const double sth = sqrt(fmax(1.0 - cth * cth, 0.0));")
                e("      double sp, cp; sincos(phi, &sp, &cp);")
                e(f"      const double q = pd{i};")
                e("      const V3 p3 = {q * sth * cp, q * sth * sp, q * cth};")
                if i == 1:
                    e(f"      {pre}b[0] = LV{{sqrt(q * q + {_f(ms[0] ** 2)}), -p3.x, -p3.y, -p3.z}};")
                    e(f"      {pre}b[1] = LV{{sqrt(q * q + {_f(ms[1] ** 2)}), p3.x, p3.y, p3.z}};")
                else:
                    e(f"      const double Esys = sqrt(q * q + Ms{i - 1} * Ms{i - 1});")
                    e("      const V3 beta = {-p3.x / Esys, -p3.y / Esys, -p3.z / Esys};")
                    for j in range(i):
                        e(f"      {pre}b[{j}] = kin_boost({pre}b[{j}], beta);")
                    e(f"      {pre}b[{i}] = LV{{sqrt(q * q + {_f(ms[i] ** 2)}), p3.x, p3.y, p3.z}};")
                e("    }")
            e(f"    w *= wl / {_f(wtmax)};")
            e("  }")
        assert draw + 2 == self.ndraw

        def place(lid, frame):
            for j, (kind, ref, _) in enumerate(levels[lid][1]):
                p = f"g{lid}_b[{j}]"
                if frame is not None:
                    p = (f"kin_boost({p}, V3{{{frame}.x / {frame}.t, {frame}.y / {frame}.t, "
                         f"{frame}.z / {frame}.t}})")
                if kind == "f":
                    e(f"  P[{ref}] = {p};")
                else:
                    e(f"  const LV g{ref}_frame = {p};")
                    place(ref, f"g{ref}_frame")

        place(0, None)
        e("  return w;")

    def source(self):
        L = [f"#define PWA_NFIN {self.nfin}", f"#define PWA_NFIELD {self.nfield}",
             f"#define PWA_NDRAW {self.ndraw}", f"#define PWA_HAS_GENBOD {int(self.ok)}"]
        body = []
        self._emit_kin(body.append)
        # F: an array of the fields, or a sink whose [] gives where one goes
        L.append("template <class Fields>\n__device__ __forceinline__ void model_kin("
                 "const LV (&P)[PWA_NFIN], Fields& F) {")
        L += body
        L.append("}\n")
        L.append("__device__ __forceinline__ double model_genbod(const double (&U)[PWA_NDRAW], "
                 "LV (&P)[PWA_NFIN]) {")
        if self.ok:
            body = []
            self._emit_genbod(body.append)
            L += body
        else:
            L.append("  return 0.0;  // masses not given: no generator")
        L.append("}\n")
        return "\n".join(L)
