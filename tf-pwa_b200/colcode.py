"""Emission of the column function: every partial-wave column of an event,
F_k,o = S_k F^ang_k,o (see ``codegen``), in one pass that hands each value to
a sink as soon as it is formed.

Chains of one topology read the same masses and angles, so what depends on
these alone is formed once per topology: the (sin, cos) of each angle that is
used at all, the phases e^{i m alpha} of the helicities that occur, q^2, its
square root and 1 / sqrt(B_l(q^2 d^2)) of each vertex.  What belongs to one
vertex at every topology (a common intermediate's decay) is formed once per
event.  D* elements keep their real d^j and their phase apart, so a real
factor costs one product instead of four; d^j_{m1 m2} is
sin^a cos^b times a homogeneous polynomial in sin^2, cos^2 of half the angle
(Horner), a = |m1 - m2|, b = |m1 + m2|.

Per vertex the barrier factor is q^l sqrt(P_l(z0) / P_l(z))
(``tf_pwa/breit_wigner.py:268-277``): 1 / sqrt(P_l(z)) is one reciprocal
square root, sqrt(P_l(z0)) a constant of the evaluation that the kernels form
once per block (``sp``, PWA_NSP values, constant pwa_sp_const[i] each).  A
Breit-Wigner with running width takes one reciprocal: with w = m P_L(q^2 d^2)
and y = Y / w, x = m0^2 - m^2, its value (x + i y) / (x^2 + y^2) is
w (x w + i Y) / ((x w)^2 + Y^2).
"""
from .particles import bprime_coeff, small_d_weight, two


def _num(v):
    r = repr(float(v))
    if "e" not in r and "." not in r and "inf" not in r and "nan" not in r:
        r += ".0"
    return r


class ColumnCode:
    """The column function of one :class:`codegen.ModelCode`."""

    def __init__(self, mc):
        self.mc = mc
        self.pairs = sorted(mc._fset)
        self.pair_index = {p: j for j, p in enumerate(self.pairs)}
        # barrier constants P_l(z0) whose square roots the kernels pass in
        self.sp = []

    # ------------------------------------------------------------ pieces
    def _sp_index(self, name):
        if name not in self.sp:
            self.sp.append(name)
        return self.sp.index(name)

    def _mass(self, chain, cf, p):
        if p in chain.inner:
            f = cf["mass"][p]
            self._use(f)
            return f"xm{f}"
        return _num(p.mass)

    def _use(self, f):
        if f not in self._loaded:
            self._loaded.append(f)

    @staticmethod
    def _tag(*parts):
        return "".join(ch if ch.isalnum() else "_" for ch in "_".join(str(p) for p in parts))

    def _inv4m2(self, out, m):
        """1 / (2 m)^2 of a mother mass: a literal, or emitted once."""
        if not m.startswith("xm"):
            return _num(0.25 / float(m) ** 2)
        nm = f"i4_{m}"
        if nm not in self._done:
            self._done.add(nm)
            out.append(f"  const double {nm} = 0.25 / ({m} * {m});")
        return nm

    def _q2(self, key):
        """Name of q^2 of a -> b c at the masses ``key`` (unclamped)."""
        nm = self._tag("q2", *key)
        out = self._scope(key)
        if nm not in self._done:
            self._done.add(nm)
            a, b, c = key
            inv = self._inv4m2(self._pass_lines if a in self._shared_mass else out, a)
            out.append(f"  const double s{nm} = {b} + {c}, d{nm} = {b} - {c};")
            out.append(f"  const double {nm} = ({a} - s{nm}) * ({a} + s{nm}) * ({a} - d{nm}) * "
                       f"({a} + d{nm}) * {inv};")
        return nm

    def _sqrt_q2(self, key):
        nm = self._q2(key)
        if "r" + nm not in self._done:
            self._done.add("r" + nm)
            self._scope(key).append(f"  const double r{nm} = sqrt({nm});")
        return "r" + nm

    def _scope(self, key):
        """Lines of the scope in which a quantity of these masses lives."""
        return self._pass_lines if key in self._shared else self._group_lines

    def _poly(self, l, z):
        co = bprime_coeff(l)
        e = _num(co[0])
        for c in co[1:]:
            e = f"fma({e}, {z}, {_num(c)})"
        return e

    def _ql(self, key, l):
        """q^l."""
        if l == 0:
            return "1.0"
        q2 = self._q2(key)
        return " * ".join(([self._sqrt_q2(key)] if l % 2 else []) + [q2] * (l // 2))

    def _barrier(self, chain, cf, d, l, out):
        """Name of the barrier factor of vertex d at l ("" when it is 1)."""
        mc = self.mc
        if not d.has_barrier_factor:
            return ""
        key = tuple(self._mass(chain, cf, p) for p in (d.core,) + tuple(d.outs))
        norm = f"{d}.norm_{l}" if d.barrier_factor_norm else None
        if l == 0 and not norm:
            return ""  # P_0 = 1
        shared = key in self._shared
        nm = self._tag("bf", mc.vertices.index(d), l, *(() if shared else (self._gid,)))
        lines = self._pass_lines if shared else out
        have = self._done if shared else self._chain_done
        if nm in have:
            return nm
        have.add(nm)
        ql = self._ql(key, l) if d.has_ql else "1.0"
        if d.has_bprime and l > 0:
            tag = self._tag(l, _num(d.d), *key)
            if "P" + tag not in self._done:
                self._done.add("P" + tag)
                sc = self._scope(key)
                z = f"({self._q2(key)} * {_num(d.d * d.d)})"
                sc.append(f"  const double P{tag} = {self._poly(l, z)};")
                sc.append(f"  const double R{tag} = prsqrt(fabs(P{tag}));")
            pz = mc.consts.index[f"{d}.Pz0_{l}"]
            i = self._sp_index(f"{d}.Pz0_{l}")
            # sqrt(P_l(z0) / P_l(z)) where that ratio is positive, else 1
            bp = f"(C.v[{pz}] * P{tag} > 0.0 ? sp[{i}] * R{tag} : 1.0)"
            bf = bp if ql == "1.0" else f"({ql}) * {bp}"
        else:
            bf = ql
        if norm:
            bf = f"({bf}) * C.v[{mc.consts.index[norm]}]"
        lines.append(f"  const double {nm} = {bf};")
        return nm

    # ------------------------------------------------------------ angles
    def _sincos(self, f, full=False):
        """(sin, cos) names of half the angle field f (of the angle: full)."""
        nm = f"{'f' if full else 'h'}{f}"
        if nm not in self._done:
            self._done.add(nm)
            self._use(f)
            x = f"xa{f}" if full else f"0.5 * xa{f}"
            self._group_lines.append(f"  double s{nm}, c{nm};")
            self._group_lines.append(f"  sincos({x}, &s{nm}, &c{nm});")
        return f"s{nm}", f"c{nm}"

    def _small_d(self, f, j2, i1, i2):
        """Expression of d^j_{m1 m2}(beta field f), i = 2 m + 2 j; "" for 1."""
        if j2 == 0:
            return ""
        w = small_d_weight(j2)
        ws = [w[l][i1 // 2][i2 // 2] for l in range(j2 + 1)]
        ls = [l for l in range(j2 + 1) if ws[l] != 0]
        if not ls:
            return "0.0"
        a, b = ls[0], j2 - ls[-1]
        n = (ls[-1] - a) // 2
        s, c = self._sincos(f)
        S, C = f"S{f}", f"C{f}"
        if n and S not in self._done:
            self._done.add(S)
            self._group_lines.append(f"  const double {S} = {s} * {s}, {C} = {c} * {c};")
        v, pw = _num(ws[a]), ""
        for k in range(1, n + 1):
            pw = S if k == 1 else f"{pw} * {S}"
            v = f"fma({v}, {C}, {_num(ws[a + 2 * k])} * {pw})"
        facs = [s] * a + [c] * b
        if n == 0 and ws[a] == 1.0 and facs:
            return " * ".join(facs)
        return " * ".join([v] + facs) if facs else v

    def _power(self, f, n):
        """(re, im) names of e^{i n x / 2} of angle field f, n > 0."""
        full = f in self._even
        if full:
            n //= 2
        s, c = self._sincos(f, full)
        base = f"{'F' if full else 'H'}{f}"
        for k in range(2, n + 1):
            nm = f"{base}_{k}"
            if nm not in self._done:
                self._done.add(nm)
                pr, pi = (c, s) if k == 2 else (f"{base}_{k - 1}r", f"{base}_{k - 1}i")
                self._group_lines.append(f"  const double {nm}r = {pr} * {c} - {pi} * {s}, "
                                         f"{nm}i = {pr} * {s} + {pi} * {c};")
        return (c, s) if n == 1 else (f"{base}_{n}r", f"{base}_{n}i")

    def _phase(self, exps):
        """(re, im, sign of im) of prod_f e^{i n_f x_f / 2}; None for 1."""
        exps = [(f, n) for f, n in sorted(exps.items()) if n]
        if not exps:
            return None
        sign = 1 if exps[0][1] > 0 else -1
        exps = [(f, sign * n) for f, n in exps]
        re, im = self._power(*exps[0])
        name = "E" + "_".join(f"{f}p{n}" if n > 0 else f"{f}m{-n}" for f, n in exps)
        if len(exps) > 1:
            if name not in self._done:
                self._done.add(name)
                for t, (f, n) in enumerate(exps[1:]):
                    a, b = self._power(f, abs(n))
                    sb = "" if n > 0 else "-"
                    last = t == len(exps) - 2
                    r2, i2 = (f"{name}r", f"{name}i") if last else (f"{name}r{t}", f"{name}i{t}")
                    self._group_lines.append(
                        f"  const double {r2} = {re} * {a} - {im} * ({sb}{b}), "
                        f"{i2} = {re} * ({sb}{b}) + {im} * {a};")
                    re, im = r2, i2
            re, im = f"{name}r", f"{name}i"
        return re, im, sign

    # ------------------------------------------------------------ lineshapes
    def _bw(self, ci, chain, cf, out):
        """(re, im) names of the chain's lineshape product, None for 1."""
        mc = self.mc
        kinds = {p: p.lineshape_kind() for p in chain.inner}
        live = [p for p in chain.inner if kinds[p] != "one"]
        if not live:
            return None
        if any(kinds[p] != "BWR" for p in live):
            for p in live:
                self._use(cf["mass"][p])
                d = chain.decay_of(p)
                for q in d.outs:
                    self._mass(chain, cf, q)
            mc._emit_lineshapes(out.append, ci)
            return f"BW_c{ci}.re", f"BW_c{ci}.im"
        res = None
        for p in live:
            d = chain.decay_of(p)
            b, c = d.outs
            m = self._mass(chain, cf, p)
            key = (m, self._mass(chain, cf, b), self._mass(chain, cf, c))
            q2, q = self._q2(key), self._sqrt_q2(key)
            L = p.bw_l if p.bw_l is not None else min(d.get_l_list())
            t = f"b{ci}_{chain.inner.index(p)}"
            ix = mc.consts.index
            # q clamped at threshold; without a q0 the width is constant in q
            out.append(f"  const bool o{t} = {m} > s{q2};")
            poly = self._poly(L, f"(z{t} * {_num(p.d * p.d)})")
            if L:
                out.append(f"  const double z{t} = o{t} ? {q2} : 0.0;")
            qp = " * ".join([q] + [q2] * L)
            out.append(f"  const double Y{t} = C.v[{ix[f'{p}.K']}] * (C.v[{ix[f'{p}.useq']}] != 0.0 "
                       f"? (o{t} ? {qp} : 0.0) : 1.0);")
            out.append(f"  const double w{t} = {m} * ({poly});")
            out.append(f"  const double x{t} = (C.v[{ix[f'{p}.m0sq']}] - {m} * {m}) * w{t};")
            out.append(f"  const double i{t} = w{t} / fma(x{t}, x{t}, Y{t} * Y{t});")
            wn = f" * C.v[{ix[f'{p}.wn']}]" if p.width_norm_applies() else ""
            out.append(f"  const double {t}r = x{t} * i{t}{wn}, {t}i = Y{t} * i{t}{wn};")
            if res is None:
                res = (f"{t}r", f"{t}i")
            else:
                out.append(f"  const double {t}R = {res[0]} * {t}r - {res[1]} * {t}i, "
                           f"{t}I = {res[0]} * {t}i + {res[1]} * {t}r;")
                res = (f"{t}R", f"{t}I")
        return res

    # ------------------------------------------------------------ chains
    def _exps(self, chain, cf, facs):
        """Phase exponents {alpha field: 2 m1} of one helicity assignment."""
        ex = {}
        for vi, i1, _, _, _ in facs:
            j2 = two(chain_vertex(chain, vi).core.J)
            if i1 != j2:
                f = cf["decays"][vi]["alpha"]
                ex[f] = ex.get(f, 0) + i1 - j2
        return ex

    def _align(self, ci, chain, cf, cur, out):
        """Contract each aligned final's helicity with D*(aligned angles)."""
        mc = self.mc
        for o, (fa, fb, fg) in cf["aligned"].items():
            oi = mc.group.outs.index(o) + 1
            j2 = two(o.J)
            new = {}
            targets = sorted({tuple(po[:oi]) + (l2,) + tuple(po[oi + 1:])
                              for po in cur for l2 in o.spins}, key=lambda t: [float(x) for x in t])
            for to in targets:
                re, im = [], []
                for l1 in o.spins:
                    src = tuple(to[:oi]) + (l1,) + tuple(to[oi + 1:])
                    if src not in cur:
                        continue
                    n1, n2 = two(l1) + j2, two(to[oi]) + j2
                    nm = f"D{oi}_{fa}_{n1}_{n2}"
                    if nm not in self._done:
                        self._done.add(nm)
                        d = self._small_d(fb, j2, n1, n2) or "1.0"
                        pr, pi, sg = self._phase({fa: n1 - j2, fg: n2 - j2}) or ("1.0", "0.0", 1)
                        self._group_lines.append(
                            f"  const double d{nm} = {d}, {nm}r = {pr} * d{nm}, "
                            f"{nm}i = {'' if sg > 0 else '-'}{pi} * d{nm};")
                    a, b = cur[src]
                    re.append(f"{a} * {nm}r" + (f" - {b} * {nm}i" if b else ""))
                    im.append(f"{a} * {nm}i" + (f" + {b} * {nm}r" if b else ""))
                self._tmp += 1
                t = f"al{self._tmp}"
                out.append(f"  const double {t}r = {' + '.join(re)}, {t}i = {' + '.join(im)};")
                new[to] = (f"{t}r", f"{t}i")
            cur = new
        return cur

    def _chain(self, ci, chain, cf, shapes):
        mc, out = self.mc, []
        self._chain_done = set()
        fac = mc._factor()
        rows = []
        for facs, po, coefs in mc.chain_assign[ci]:
            ds = []
            for vi, i1, i2, _, _ in facs:
                d = self._small_d(cf["decays"][vi]["beta"], two(chain_vertex(chain, vi).core.J), i1, i2)
                if d:
                    ds.append(d)
            if any(d == "0.0" for d in ds):
                continue
            ph = self._phase(self._exps(chain, cf, facs))
            t = f"t{ci}_{len(rows)}"
            out.append(f"  const double {t} = {' * '.join(f'({d})' for d in ds) if ds else '1.0'};")
            im = None
            re = t
            if ph is not None:
                out.append(f"  const double {t}r = {t} * {ph[0]}, "
                           f"{t}i = {t} * {'' if ph[2] > 0 else '-'}{ph[1]};")
                re, im = f"{t}r", f"{t}i"
            rows.append((po, coefs, re, im))
        bw = self._bw(ci, chain, cf, out) if shapes else None
        for k in mc.chain_columns[ci]:
            sums = {}
            for po, coefs, re, im in rows:
                if k in coefs:
                    r, i = sums.setdefault(po, ([], []))
                    r.append((coefs[k], re))
                    if im:
                        i.append((coefs[k], im))
            cur = {}
            for po, (r, i) in sums.items():
                self._tmp += 1
                t = f"F{self._tmp}"
                out.append(f"  const double {t}r = {self._dot(r)};")
                if i:
                    out.append(f"  const double {t}i = {self._dot(i)};")
                cur[po] = (f"{t}r", f"{t}i" if i else "")
            cur = self._align(ci, chain, cf, cur, out)
            lsi = mc.columns[k][1]
            bfs = [self._barrier(chain, cf, d, d.get_ls_list()[lsi[vi]][0], out)
                   for vi, d in enumerate(chain)]
            sc = [b for b in bfs if b] + ([_num(fac)] if fac != 1.0 else [])
            sc = " * ".join(sc) if sc else "1.0"
            self._tmp += 1
            S = f"S{self._tmp}"
            if bw is None:
                out.append(f"  const double {S} = {sc};")
            else:
                out.append(f"  const double {S} = {sc}, {S}r = {bw[0]} * {S}, {S}i = {bw[1]} * {S};")
            for po, (a, b) in cur.items():
                o = mc._out(po)
                j = self.pair_index[(k, o)]
                if bw is None:
                    v = f"{S} * {a}, {f'{S} * {b}' if b else '0.0'}"
                elif b:
                    v = f"{S}r * {a} - {S}i * {b}, {S}r * {b} + {S}i * {a}"
                else:
                    v = f"{S}r * {a}, {S}i * {a}"
                verb = "add" if (k, o) in self._written else "set"
                self._written.add((k, o))
                out.append(f"  F.{verb}({k}, {o}, {j}, {v});")
        return out

    @staticmethod
    def _dot(terms):
        e = ""
        for c, x in terms:
            c = f"(cc ? {_num(c[1])} : {_num(c[0])})" if isinstance(c, tuple) else _num(c)
            if not e:
                e = x if c == "1.0" else f"-{x}" if c == "-1.0" else f"{c} * {x}"
            else:
                e = f"fma({c}, {x}, {e})"
        return e

    # ------------------------------------------------------------ function
    def _geometry(self, ci, cf):
        mc = self.mc
        return (tuple((a["alpha"], a["beta"]) for a in cf["decays"]),
                tuple((mc.group.outs.index(o),) + tuple(v) for o, v in cf["aligned"].items()))

    def body(self, shapes):
        """Lines of the function body (loads first)."""
        mc = self.mc
        self._loaded, self._written, self._tmp = [], set(), 0
        lines = []
        for ps in range(mc.npass):
            mc._pass = ps
            groups = {}
            for ci, c in enumerate(mc.group):
                groups.setdefault(self._geometry(ci, mc._cf(ci)), []).append(ci)
            # vertices (at their masses) that several groups share
            keys, seen, masses = {}, [], {}
            for gi, cis in enumerate(groups.values()):
                for ci in cis:
                    cf, c = mc._cf(ci), mc.group[ci]
                    for d in c:
                        key = tuple(self._mass(c, cf, p) for p in (d.core,) + tuple(d.outs))
                        keys.setdefault(key, set()).add(gi)
                        masses.setdefault(key[0], set()).add(gi)
            self._shared = {k for k, g in keys.items() if len(g) > 1}
            self._shared_mass = {m for m, g in masses.items() if len(g) > 1 and m.startswith("xm")}
            self._done = set()
            self._pass_lines = []
            body = []
            for gi, cis in enumerate(groups.values()):
                self._gid = gi
                self._group_lines = []
                # names of an earlier group's scope are gone
                keep = set(self._done)
                exps = {}
                for ci in cis:
                    cf, c = mc._cf(ci), mc.group[ci]
                    for facs, _, _ in mc.chain_assign[ci]:
                        for f, n in self._exps(c, cf, facs).items():
                            exps.setdefault(f, set()).add(n)
                    for o, (fa, _, fg) in cf["aligned"].items():
                        for f in (fa, fg):
                            exps.setdefault(f, set()).update(two(s) for s in o.spins)
                self._even = {f for f, ns in exps.items() if all(n % 2 == 0 for n in ns)}
                chains = []
                for ci in cis:
                    chains.append((ci, self._chain(ci, mc.group[ci], mc._cf(ci), shapes)))
                body.append(f"  {{ // topology {gi}" + (f" (swap {ps})" if ps else ""))
                body += self._group_lines
                for ci, ls in chains:
                    body.append(f"  {{ // chain {ci}: {mc.group[ci]}")
                    body += ls
                    body.append("  }")
                body.append("  }")
                # keep what went to the pass scope, forget the group's names
                shared_text = "\n".join(self._pass_lines)
                self._done = {n for n in self._done if n in keep or self._declared(n, shared_text)}
            lines.append("  {")
            lines += self._pass_lines + body
            lines.append("  }")
        mc._pass = 0
        # every structural pair is written
        lines += [f"  F.set({k}, {o}, {j}, 0.0, 0.0);" for j, (k, o) in enumerate(self.pairs)
                  if (k, o) not in self._written]
        head = []
        for f in sorted(self._loaded):
            if f in mc.mass_slot:
                a = f"XM + (long long){mc.mass_slot[f]} * ld + i"
                head.append(f"  const double xm{f} = LDG ? __ldg({a}) : *({a});")
            else:
                a = f"XA + (long long){mc.angle_slot[f]} * ld + i"
                head.append(f"  const double xa{f} = LDG ? __ldg({a}) : *({a});")
        if mc.flips:
            ci = mc.plan.charge_index
            if ci not in self._loaded:
                a = f"XM + (long long){mc.mass_slot[ci]} * ld + i"
                head.append(f"  const double xm{ci} = LDG ? __ldg({a}) : *({a});")
            head.append(f"  const bool cc = xm{ci} < 0.0;")
            head.append("  (void)cc;")
        return head + lines

    @staticmethod
    def _declared(name, text):
        return f"const double {name} =" in text or f", {name} =" in text

    def source(self):
        """``model_cols`` (with the lineshapes) and ``model_cols_ns``
        (without), and the wrappers that fill a dense array."""
        L = []
        parts = [(name, self.body(shapes)) for name, shapes in (("model_cols", True),
                                                                ("model_cols_ns", False))]
        n = max(len(self.sp), 1)
        idx = [self.mc.consts.index[s] for s in self.sp] or [0]
        L.append(f"#define PWA_NPASS {self.mc.npass}")
        L.append(f"#define PWA_NSP {n}")
        L.append("__device__ constexpr int pwa_sp_const[PWA_NSP] = {" + ", ".join(map(str, idx)) + "};")
        for name, body in parts:
            L.append(f"template <bool LDG, class Sink>\n__device__ __forceinline__ void {name}(\n"
                     "    const Consts& C, const double* __restrict__ sp, const double* __restrict__ XA,\n"
                     "    const double* __restrict__ XM, long long ld, long long i, Sink& F) {\n"
                     "  using R = double;")
            L += body
            L.append("}\n")
        L.append("""// the columns as a dense array F[k * PWA_NOUT + o], zero where a pair has no
// structural value
struct DenseColumns {
  cpx<double>* f;
  __device__ __forceinline__ void set(int k, int o, int, double re, double im) {
    f[k * PWA_NOUT + o] = cmk<double>(re, im);
  }
  __device__ __forceinline__ void add(int k, int o, int, double re, double im) {
    f[k * PWA_NOUT + o].re += re;
    f[k * PWA_NOUT + o].im += im;
  }
};""")
        for wrap, name in (("model_columns", "model_cols"), ("model_columns_ns", "model_cols_ns")):
            fn = (f"template <typename R, bool LDG = true>\n__device__ __forceinline__ void {wrap}(\n"
                  "    const Consts& C, const R* __restrict__ XA, const double* __restrict__ XM,\n"
                  "    long long ld, long long i, cpx<R>* __restrict__ F) {\n"
                  "  double sp[PWA_NSP];\n"
                  "  for (int j = 0; j < PWA_NSP; ++j) sp[j] = sqrt(fabs(C.v[pwa_sp_const[j]]));\n"
                  "  for (int j = 0; j < PWA_NCOL * PWA_NOUT; ++j) F[j] = cmk<R>(R(0), R(0));\n"
                  "  DenseColumns s{F};\n"
                  f"  {name}<LDG>(C, sp, XA, XM, ld, i, s);\n"
                  "}\n")
            # the kernels take the shape-free columns through sinks of their own
            L.append(fn if wrap == "model_columns" else f"#ifndef __CUDACC__\n{fn}#endif\n")
        return "\n".join(L)


def chain_vertex(chain, vi):
    return list(chain)[vi]
