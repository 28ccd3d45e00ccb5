"""FP64 ERI kernels: one warp (or more) per contracted quartet.

Two bodies inside one frame (WarpEmitter).  ThreadEmitter runs the Obara-Saika
recurrences of a primitive quartet in one lane, for classes with few targets;
RysEmitter evaluates the others by Rys quadrature:

[e0|f0] = sum over the N = L/2 + 1 roots of I_x(e_x, f_x) I_y(e_y, f_y) I_z(e_z, f_z),
with the 2D integrals of each root and axis from the recurrences
  I(0, 0) = 1 (z axis: the weight times the prefactor)
  I(e + 1, f) = C I(e, f) + e B10 I(e - 1, f) + f B00 I(e, f - 1)
  I(e, f + 1) = D I(e, f) + f B01 I(e, f - 1) + e B00 I(e - 1, f)
(Rys, Dupuis, King, J. Comput. Chem. 4, 154 (1983)).  Per chunk of primitive
quartets a warp runs four steps, each with its lanes over other work items:

  setup    lane = primitive quartet: pair data from the lists in shared memory,
           geometry, Boys argument
  roots    lane = (primitive quartet, root): table polynomials (rys_table.py)
  2D       lane = (primitive quartet, root, axis): the (S+1)(C+1) integrals of
           its axis, into shared memory
  product  lane = (primitive quartet, target component s of the lane side): for
           every root the 3 (C+1) integrals of s, then the products for every
           target c of the chain side, added to the accumulators in registers

Only the target levels la..la+lb and lc..lc+ld get lanes and accumulators, no
lane evaluates a value twice, and nothing is exchanged between dependent
recurrence levels.  Several primitive quartets share a warp in the product step
(QPW = 32 // targets); lane sides of more than 32 targets take several warps, and
chain sides of more than MAX_ACC targets are split over warps as well.

What bounds them (B200, FP64): the large classes' product step, its shared loads
(69-76 % of the load/store unit's cycles on (dp|dp) and (dd|dd); every lane reads
its own 3 (C + 1) integrals of a root, so a wider chain side is read less often
per product: plan() weighs the two), the classes with few primitive quartets
latency at 12-16 warps an SM.  ns per quartet, K 1..6 in a 30-bohr box, against
the lane-group kernels of the recurrences (group_emitter.py) that these replace:
(ss|ss) 8.1 -> 2.9, (ps|ps) 10.5 -> 3.7, (pp|ps) 12.5 -> 5.1, (dp|dp) 55 -> 28,
(dd|dd) 110 -> 56, (fd|dd) 297 -> 170, (ff|dd) 1082 -> 785; (ff|ff) is level (1.9 us).
With few primitives (s shells of 3 or 6, p of 3, d and f of one, 8 bohr):
(ss|ss) 12.7 -> 4.1, (dd|dd) 16.1 -> 8.5, (ff|dd) 48 -> 33, but (ds|ds) 4.1 -> 5.2 and
(dd|ds) 6.3 -> 7.6: ten-lane groups put three such quartets in a warp, a warp
here holds one.  Quartets of so few primitive quartets keep the lane-group
kernels in large batches (eri_emitter.SHORT).
"""
from intception_b200.basis import sph_matrix

from .eri_emitter import ZERO, Emitter, class_id, comps, comps_range
from .group_emitter import GroupEmitter, MINB_VALUES, ncart, ncum

CHUNK = 32      # primitive quartets per setup step
PAIR_TILE = 64  # live pairs per side and tile
MAX_ACC = 81    # accumulators per lane (162 registers)


def pairs_targets(l0, l1):
    return comps_range(l0, l0 + l1)


def plan(la, lb, lc, ld):
    """Geometry of the class's kernel: orient ('bra': lanes own bra targets), NS lane targets, parts of the chain
    side, G lanes per group, QPW primitive quartets per product step."""
    best = None
    for orient in ('bra', 'ket'):
        (s0, s1), (c0, c1) = ((la, lb), (lc, ld)) if orient == 'bra' else ((lc, ld), (la, lb))
        NS, NC = len(pairs_targets(s0, s1)), len(pairs_targets(c0, c1))
        parts = 1
        while -(-NC // parts) > MAX_ACC:
            parts *= 2
        warps = -(-NS // 32) * parts
        QPW = 32 // NS if NS <= 16 else 1
        C = c0 + c1
        # shared loads (2 cycles each, one port) or FP64 (2 cycles on each of four ports) per primitive quartet
        nxy = (C + 1) * (C + 2) // 2
        cost = warps * max(6.0 * (C + 1), 0.5 * (nxy + NC)) / QPW
        if best is None or cost < best[0]:
            best = (cost, orient, NS, parts, 32 * warps, QPW)
    return dict(orient=best[1], NS=best[2], parts=best[3], G=best[4], QPW=best[5])


class WarpEmitter(GroupEmitter):
    """The frame that both kernels share: quartet assignment, pair lists and
    pair data in shared memory, chunks of primitive quartets, the sum of the
    slices, the HRR check and the epilogue (GroupEmitter's)."""

    G = 32  # lanes per group
    chunk = CHUNK

    def __init__(self, la, lb, lc, ld):
        # no GroupEmitter layout: only its epilogue pieces are used
        self.la, self.lb, self.lc, self.ld = la, lb, lc, ld
        self.L, self.E, self.F = la + lb + lc + ld, la + lb, lc + ld
        self.tag = '%d%d%d%d' % (la, lb, lc, ld)
        self.cid = class_id(la, lb, lc, ld)

    @property
    def name(self):
        return 'ib_%s_%s' % (self.kind, self.tag)

    def quartet_code(self, stride=None):
        """Code of one quartet (item *itp, sorted index p) on its lanes: the
        declarations that depend on the lane only, and the evaluation.
        stride: doubles of shared memory between groups (default: the class's
        own need; a kernel of several classes gives them one stride, as their
        groups lie side by side)."""
        G = self.G
        # threads per block: four warps, or one group where that is not a part of them
        self.block = 128 if G in (32, 64, 128) else G
        wide = G > 32
        NE, NF = ncum(self.E) - ncum(self.la - 1), ncum(self.F) - ncum(self.lc - 1)
        NFP = NF if NF % 2 else NF + 1
        TBL = NE * NFP
        epi_cart, sm_cart = self.emit_epilogue(False)
        epi_sph, sm_sph = self.emit_epilogue(True)
        area, ntab = self.layout(TBL)
        area = max(area, sm_cart, sm_sph)
        # then (slice 0): pair data, pair lists and screening exponents, counts, screened queue
        o_pair = area + (area & 1)
        o_lst = o_pair + 2 * PAIR_TILE * 4
        o_cnt = o_lst + 32
        o_que = o_cnt + 2
        per_group = o_que + 2 * CHUNK // 4 + 2
        per_group += per_group & 1
        self.smem = 8 * (self.block // G) * per_group
        self.per_group = per_group
        if stride is not None:
            assert stride >= per_group
            per_group = stride
        NB = getattr(self, 'NB', 1)
        sync = 'ib_group_bar(gid, %d)' % G if wide else '__syncwarp()'
        src = []
        A = src.append
        A('  const unsigned sgmask = 0xffffffffu;')
        A('  const int sg = gid / W, w = gid - sg * W;  // quartet slot in the block, slice in the quartet')
        A('  const int SG = W * %d, r = w * %d + j;  // lanes per quartet, this lane among them' % (G, G))
        A('  double* __restrict__ sb = ib_smem + gid * %d;' % per_group)
        A('  double* __restrict__ sb0 = ib_smem + sg * W * %d;  // slice 0' % per_group)
        A('  unsigned char* __restrict__ lst = reinterpret_cast<unsigned char*>(sb0 + %d);' % o_lst)
        A('  int* __restrict__ lcnt = reinterpret_cast<int*>(sb0 + %d);' % o_cnt)
        A('  unsigned short* __restrict__ que = reinterpret_cast<unsigned short*>(sb + %d);' % o_que)
        if wide:
            A('  int* __restrict__ qcnt = reinterpret_cast<int*>(sb + %d);' % (per_group - 2))
        A('  double* __restrict__ pd = sb0 + %d;' % o_pair)
        src += self.prologue()
        head, src = src, []
        A = src.append
        A('    IbQuartet g;')
        A('    ib_load_quartet(a, *itp, g);')
        A('    const int kb_ = g.k[1], kd_ = g.k[3];')
        A('    const int kab = g.k[0] * kb_, kcd = g.k[2] * kd_;')
        # classes with a g shell build only the exact-zero lists: skipping
        # primitive quartets is allowed, not asked for, and the screened lists
        # were never measured there
        if max(self.la, self.lb, self.lc, self.ld) >= 4:
            A('    constexpr bool pre = false;  // g classes: exact-zero lists only')
        else:
            A('    const bool pre = a.prim_tol > 0.0 && kab <= 64 && kcd <= 64;  // uniform over the quartet')
        A('    if (pre && r < 32) {')
        A('      const int2 nn = ib_live_pairs_screened<%s, SPH>(a.prim_exp, a.prim_coef, g.ptr[0], g.ptr[1], '
          'kb_, g.ptr[2], g.ptr[3], kd_, g.RAB2, g.RCD2, 0, kab, 0, kcd, lst, r, 32, 0xffffffffu, 0, a.prim_tol);'
          % self.lcls())
        A('      __syncwarp();')
        A('      for (int x = r; x < nn.x; x += 32) ib_pair_data(a, g, 0, lst[x], pd + 4 * x);')
        A('      for (int x = r; x < nn.y; x += 32) ib_pair_data(a, g, 1, lst[64 + x], pd + 4 * (%d + x));' % PAIR_TILE)
        A('      if (r == 0) { lcnt[0] = nn.x; lcnt[1] = nn.y; }')
        A('    }')
        A('    double acc[%d];' % self.nacc())
        A('#pragma unroll')
        A('    for (int k = 0; k < %d; ++k) acc[k] = 0.0;' % self.nacc())
        A('    for (int ab0 = 0; ab0 < kab; ab0 += %d)' % PAIR_TILE)
        A('    for (int cd0 = 0; cd0 < kcd; cd0 += %d) {' % PAIR_TILE)
        A('      if (r < 32 && !pre) {')
        A('        const int n0 = ib_live_pair_data(a, g, 0, ab0, min(%d, kab - ab0), pd, r);' % PAIR_TILE)
        A('        const int n1 = ib_live_pair_data(a, g, 1, cd0, min(%d, kcd - cd0), pd + %d, r);'
          % (PAIR_TILE, 4 * PAIR_TILE))
        A('        if (r == 0) { lcnt[0] = n0; lcnt[1] = n1; }')
        A('      }')
        A('      ib_sg_sync(SG, sg, sgmask);')
        A('      const int nl1 = lcnt[1], npl = lcnt[0] * nl1;')
        A('      const float rn1 = 1.0f / (float)max(nl1, 1);')
        # chunks of the unscreened loop: as even over the slices as the 2D step allows
        if NB > 1:
            A('      const int ch = min(%d, ((npl + W - 1) / W + %d) / %d * %d);' % (self.chunk, NB - 1, NB, NB))
        else:
            A('      const int ch = min(%d, max((npl + W - 1) / W, 1));' % CHUNK)
        A('      int q0 = pre ? 32 * w : ch * w, left = 0;')
        A('      while (true) {')
        A('        int n, qa = 0, qc = 0;  // primitive quartets of this chunk; the lane\'s list positions')
        A('        if (pre) {')
        # survivors of the screen, collected by the group's first warp
        A('          if (j < 32) {')
        A('            while (left < %d && q0 < npl) {' % self.chunk)
        A('              const int u = q0 + j, ua = (int)(((float)u + 0.5f) * rn1), uc = u - ua * nl1;')
        A('              const bool ok = u < npl && !ib_quartet_negligible(lst, ua, uc, a.prim_tol);')
        A('              const unsigned bal = __ballot_sync(0xffffffffu, ok);')
        A('              if (ok) que[left + __popc(bal & ((1u << j) - 1u))] = (unsigned short)(ua | (uc << 8));')
        A('              left += __popc(bal);')
        A('              q0 += 32 * W;')
        A('            }')
        if wide:
            A('            if (j == 0) *qcnt = left;')
        A('          }')
        A('          %s;' % sync)
        A('          n = min(%s, %d);' % ('*qcnt' if wide else 'left', self.chunk))
        A('          if (n == 0) break;  // uniform over the group')
        A('          if (j < n) { qa = que[j] & 255; qc = que[j] >> 8; }')
        A('        } else {')
        A('          if (q0 >= npl) break;')
        A('          n = min(ch, npl - q0);')
        A('          const int u = q0 + j;')
        A('          qa = (int)(((float)u + 0.5f) * rn1);')
        A('          qc = u - qa * nl1;')
        A('          q0 += ch * W;')
        A('        }')
        src += self.chunk_body(sync)
        A('        %s;  // the chunk\'s shared data are free' % sync)
        A('        if (pre && j < 32) {  // survivors past this chunk move to the front')
        A('          left -= n;')
        A('          const unsigned short v = j < left ? que[n + j] : (unsigned short)0;')
        A('          __syncwarp();')
        A('          if (j < left) que[j] = v;')
        A('          __syncwarp();')
        A('        }')
        A('      }')
        A('      ib_sg_sync(SG, sg, sgmask);  // every slice is done with the lists before the next tile')
        A('    }')
        src += self.write_tables(NFP, TBL)
        A('    ib_sg_sync(SG, sg, sgmask);')
        A('    if (W * %d > 1) {  // sum of the partial tables' % ntab)
        A('      for (int x = r; x < %d; x += SG) {' % (NE * NF))
        A('        const int o = (x / %d) * %d + x %% %d;' % (NF, NFP, NF))
        A('        double s = 0.0;')
        A('        for (int v = 0; v < W; ++v)')
        A('#pragma unroll')
        A('          for (int k = 0; k < %d; ++k) s += sb0[v * %d + k * %d + o];' % (ntab, per_group, TBL))
        A('        sb0[o] = s;')
        A('      }')
        A('      ib_sg_sync(SG, sg, sgmask);')
        A('    }')
        if self.lb or self.ld:
            src += self.hrr_check(NE, NF, NFP)
        A('    const double ABx = g.AB[0], ABy = g.AB[1], ABz = g.AB[2];')
        A('    const double CDx = g.CD[0], CDy = g.CD[1], CDz = g.CD[2];')
        A('    (void)ABx; (void)ABy; (void)ABz; (void)CDx; (void)CDy; (void)CDz;')
        A('    double* __restrict__ o = a.out + g.off;')
        A('    if (SPH) {')
        src += ['  ' + s for s in epi_sph]
        A('    } else {')
        src += ['  ' + s for s in epi_cart]
        A('    }')
        A('    ib_sg_sync(SG, sg, sgmask);')
        return head, src

    def kernel(self):
        """CUDA source of the class's FP64 kernel: its groups take the quartets
        of the class's range one at a time."""
        head, body = self.quartet_code()
        src = ['// ---- class (%d%d|%d%d): %s' % (self.la, self.lb, self.lc, self.ld, self.describe())]
        src += self.constants()
        src += ['template <bool SPH, int MINB>',
                '__global__ void __launch_bounds__(%d, MINB) %s(const IbLaunch a) {' % (self.block, self.name),
                '  extern __shared__ double ib_smem[];',
                '  constexpr int GPB = %d;  // groups per block' % (self.block // self.G),
                '  const int beg = a.ranges[2 * %d], end = a.ranges[2 * %d + 1];' % (self.cid, self.cid),
                '  const int W = ib_slices(end - beg, GPB, a.max_slices, a.slice_boost);',
                '  const int SPB = GPB / W;  // quartets in flight per block',
                '  if (beg + (int)blockIdx.x * SPB >= end) return;  // block-uniform',
                '  const int gid = threadIdx.x / %d, j = threadIdx.x %% %d;' % (self.G, self.G)]
        src += head
        grab = 'ib_grab(a.counter, beg, r, SG, sg, sgmask, 0, lcnt + 2)'
        src += ['  for (int p = %s; p < end; p = %s) {' % (grab, grab),
                '    if (a.recheck && !(a.flags[p] & 1)) continue;  // uniform over the quartet\'s lanes',
                '    const IbItem* __restrict__ itp = a.items + p;']
        return '\n'.join(src + body + ['  }', '}', ''])

    def function(self, stride):
        """The same evaluation as a device function of one quartet, for the
        small-batch kernel (G = 32: one to four warps a quartet)."""
        assert self.G == 32
        head, body = self.quartet_code(stride)
        src = self.constants()
        src += ['template <bool SPH>',
                '__device__ __noinline__ void %s_one(const IbLaunch& a, const IbItem* itp, int p, int W) {' % self.name,
                '  extern __shared__ double ib_smem[];',
                '  const int gid = threadIdx.x / 32, j = threadIdx.x % 32;']
        return '\n'.join(src + head + ['  (void)lcnt; (void)que;'] + body + ['}', ''])

    def split_bra(self):
        # measured as instructions of one warp: a whole bra recurrence per f
        # (about 9 an output) in ceil(NF/32) rounds, against about 60 and 30 an
        # (f, a) and (f, b) item
        NF = ncum(self.F) - ncum(self.lc - 1)
        return NF <= 16 and self.la >= 1

    def emit_bra_split(self, sph, NF, NFP, L):
        """Bra HRR with lanes over (f, a): each lane raises b for its own a (the
        component index of a + k is that of a plus a constant and |k_y + k_z|
        times a_y + a_z), transforms b, and lanes over (f, b) then transform a.
        Returns the offset of the [ab][f] table and the doubles used."""
        la, lb = self.la, self.lb
        NA, NB = ncart(la), (2 * lb + 1) if sph else ncart(lb)
        NE = ncum(self.E) - ncum(la - 1)
        B1 = NE * NFP
        cur, size = 0, B1
        if lb or (sph and la == 1):
            # spherical p functions m = -1, 0, 1 are y, z, x
            row = '((av + 2) % 3)' if sph and la == 1 else 'av'
            L.append('    for (int x = r; x < %d; x += SG) {' % (NF * NA))
            L.append('      const int av = x / %d, t = x - av * %d;' % (NF, NF))
            L.append('      const int s = %s;' % (' + '.join('(av >= %d)' % (k * (k + 1) // 2) for k in range(1, la + 1))))
            L.append('      const double* __restrict__ q = sb0 + av * %d + t;' % NFP)
            L.append('      const int sn = s * %d; (void)sn;' % NFP)
            names, body, cnt = {}, [], [0]

            def leaf(k):
                if k not in names:
                    ks = k[1] + k[2]
                    c = ncum(la + sum(k) - 1) - ncum(la - 1) + k[2] + ks * (ks + 1) // 2
                    names[k] = 'q%d_%d_%d' % k
                    body.append('      const double %s = q[%d%s];' % (names[k], c * NFP, ' + %d * sn' % ks if ks else ''))
                return names[k]
            res = self._hrr([ZERO], comps(lb), leaf, 'AB', 'h', body, cnt)
            vals = [res[(ZERO, b)] for b in comps(lb)]
            L += body
            if sph:
                vals = self._sph1(vals, lb, 'tb', L)
            for i, v in enumerate(vals):
                L.append('      sb0[%d + (%s * %d + %d) * %d + t] = %s;' % (B1, row, NB, i, NFP, v))
            L += ['    }', '    ib_sg_sync(SG, sg, sgmask);']
            cur, size = B1, B1 + NA * NB * NFP
        if sph and la >= 2:
            dst = 0 if cur else B1
            L.append('    for (int x = r; x < %d; x += SG) {' % (NF * NB))
            L.append('      const int bv = x / %d, t = x - bv * %d;' % (NF, NF))
            for i in range(NA):
                L.append('      const double c%d = sb0[%d + (%d + bv) * %d + t];' % (i, cur, i * NB, NFP))
            for i, v in enumerate(self._sph1(['c%d' % i for i in range(NA)], la, 'ta', L)):
                L.append('      sb0[%d + (%d + bv) * %d + t] = %s;' % (dst, i * NB, NFP, v))
            L += ['    }', '    ib_sg_sync(SG, sg, sgmask);']
            size = max(size, dst + (2 * la + 1) * NB * NFP)
            cur = dst
        return cur, size

    @staticmethod
    def _sph1(vals, l, prefix, lines):
        """Cartesian values of one index -> spherical names."""
        T = sph_matrix(l)
        out = []
        for s in range(2 * l + 1):
            terms = [vals[i] if abs(T[i, s] - 1) < 1e-15 else '%.17g * %s' % (T[i, s], vals[i])
                     for i in range(len(vals)) if abs(T[i, s]) > 1e-15]
            lines.append('      const double %s%d = %s;' % (prefix, s, ' + '.join(terms)))
            out.append('%s%d' % (prefix, s))
        return out

    def budget(self):
        """Register budget (index into MINB_VALUES): the most resident blocks
        whose registers hold the accumulators, the values in flight and some
        forty more, and whose shared memory fits."""
        need = 2 * self.nacc() + self.in_flight() + 44
        best = 0
        for mi, minb in enumerate(MINB_VALUES):
            per_part = -(-minb * self.block // 32 // 4)  # warps of an SM quarter, which shares 16384 registers
            if 512 // per_part >= need and minb * (self.smem + 1024) <= 227 * 1024:
                best = mi
        return best


class RysEmitter(WarpEmitter):
    kind = 'rys'

    def __init__(self, la, lb, lc, ld):
        super().__init__(la, lb, lc, ld)
        self.N = self.L // 2 + 1
        p = plan(la, lb, lc, ld)
        self.orient, self.NS, self.parts, self.G, self.QPW = p['orient'], p['NS'], p['parts'], p['G'], p['QPW']
        self.bra = self.orient == 'bra'
        if self.bra:
            self.S, self.S_lo, self.C, self.C_lo = self.E, la, self.F, lc
        else:
            self.S, self.S_lo, self.C, self.C_lo = self.F, lc, self.E, la
        self.stargets = comps_range(self.S_lo, self.S)
        self.ctargets = comps_range(self.C_lo, self.C)
        self.NC = len(self.ctargets)
        # doubles per (root, axis) table, odd so that lanes writing consecutive tables hit all banks
        self.TS = (self.S + 1) * (self.C + 1)
        self.TS += 1 - self.TS % 2
        # primitive quartets per 2D step: a multiple of QPW that fills the lanes
        # of its tasks well, within 8 KB a warp
        best = None
        for k in range(1, 9):
            nb = k * self.QPW
            if nb > CHUNK or (k > 1 and nb * 3 * self.N * self.TS > 1024 * (self.G // 32)):
                break
            tasks = nb * 3 * self.N
            waste = -(-tasks // self.G) * self.G / tasks
            if best is None or waste < best[0] - 0.05:
                best = (waste, nb)
        self.NB = best[1]
        self.PS = self.prim_stride()

    def prim_stride(self):
        """Doubles between the tables of two primitive quartets, padded so that
        the product step's half-warp loads collide least."""
        base = 3 * self.N * self.TS
        if self.QPW == 1:
            return base
        best = None
        for pad in range(16):
            worst = 0
            for axis in range(3):
                for half in (0, 16):
                    addr = set()
                    for lane in range(half, half + 16):
                        g, s = divmod(lane, self.NS)
                        if g < self.QPW:
                            addr.add(g * (base + pad) + self.stargets[s][axis] * (self.C + 1))
                    hits = {}
                    for a in addr:
                        hits[a % 16] = hits.get(a % 16, 0) + 1
                    worst += max(hits.values()) if hits else 0
            if best is None or worst < best[0]:
                best = (worst, pad)
        return base + best[1]

    # ------------------------------------------------------------- pieces
    def chain_code(self):
        """2D integrals of one (primitive quartet, root, axis), axis d, stored at tb[s * (C + 1) + c]."""
        S, C = self.S, self.C
        L = []
        if self.bra:
            L += ['          const double SX = Cx, CX = Dx, SB = B10, CB = B01;']
        else:
            L += ['          const double SX = Dx, CX = Cx, SB = B01, CB = B10;']
        L.append('          (void)SX; (void)CX; (void)SB; (void)CB;')
        v = {}

        def put(s, c, expr):
            if expr is not None:
                L.append('          const double i%d_%d = %s;' % (s, c, expr))
            v[s, c] = 'i%d_%d' % (s, c)
            L.append('          tb[%d] = i%d_%d;' % (s * (C + 1) + c, s, c))

        def mul(k, name):
            return name if k == 1 else '%d.0 * %s' % (k, name)
        for k in range(2, max(S, C) + 1):
            if k <= S:
                L.append('          const double nB00_%d = %d.0 * B00; (void)nB00_%d;' % (k, k, k))
        nb00 = lambda k: 'B00' if k == 1 else 'nB00_%d' % k  # noqa: E731
        put(0, 0, 'd == 2 ? wt : 1.0')
        for s in range(S):
            e = 'SX * i%d_0' % s
            if s:
                e = 'fma(SX, i%d_0, (%s) * i%d_0)' % (s, mul(s, 'SB'), s - 1)
            put(s + 1, 0, e)
        for c in range(C):
            for s in range(S + 1):
                e = 'CX * i%d_%d' % (s, c)
                if c:
                    e = 'fma(CX, i%d_%d, (%s) * i%d_%d)' % (s, c, mul(c, 'CB'), s, c - 1)
                if s:
                    e = 'fma(%s, i%d_%d, %s)' % (nb00(s), s - 1, c, e)
                put(s, c + 1, e)
        return L

    def product_code(self, part):
        """Products of one root for the chain targets of part; loads at tx, ty, tz."""
        C = self.C
        tg = self.part_targets(part)
        idx = {c: t for t, c in enumerate(tg)}
        L = []
        need_y = sorted({c[1] for c in tg})
        need_z = sorted({c[2] for c in tg})
        for k in need_z:
            L.append('            const double z%d = tz[%d];' % (k, k))
        for k in need_y:
            L.append('            const double y%d = ty[%d];' % (k, k))
        for cx in range(C + 1):
            use = [c for c in tg if c[0] == cx]
            if not use:
                continue
            L.append('            const double x%d = tx[%d];' % (cx, cx))
            for cy in sorted({c[1] for c in use}):
                L.append('            const double p%d_%d = x%d * y%d;' % (cx, cy, cx, cy))
                for c in use:
                    if c[1] == cy:
                        L.append('            acc[%d] = fma(p%d_%d, z%d, acc[%d]);' % (idx[c], cx, cy, c[2], idx[c]))
        return L

    def part_targets(self, part):
        """Chain targets of one part: contiguous runs of the (level-ordered) list."""
        n = -(-self.NC // self.parts)
        return self.ctargets[part * n:(part + 1) * n]

    # ------------------------------------------------------------- bodies
    def layout(self, tbl):
        """Shared memory of a group, in doubles: setup fields, roots and
        weights, 2D tables; the contracted tables take the same area afterwards."""
        self.o_uw = 12 * CHUNK
        self.o_tab = self.o_uw + 2 * self.N * CHUNK
        return max(self.o_tab + self.NB * self.PS, self.QPW * tbl), self.QPW

    def in_flight(self):
        return 2 * (2 * (self.C + 1) + 3)

    def nacc(self):
        return max(len(self.part_targets(h)) for h in range(self.parts))

    def prologue(self):
        NS, QPW, TS, PS, C = self.NS, self.QPW, self.TS, self.PS, self.C
        W32 = self.G // 32 // self.parts  # warps over the lane targets
        L = []
        if self.parts > 1:
            L += ['  const int part = j / %d;' % (32 * W32), '  const int jj = j %% %d;' % (32 * W32)]
        else:
            L += ['  const int jj = j;']
        if QPW > 1:
            L += ['  const int pg = jj / %d, js = jj %% %d;  // primitive quartet of the step, lane target' % (NS, NS),
                  '  const bool own = pg < %d;' % QPW]
        else:
            L += ['  constexpr int pg = 0;', '  const int js = jj;', '  const bool own = jj < %d;' % NS]
        L.append('  const unsigned code = ib_pin(own ? ib_rlane_%s[js] : 0);' % self.tag)
        for axis, name, sh in ((0, 'ptx', 'code & 15u'), (1, 'pty', '(code >> 4) & 15u'), (2, 'ptz', '(code >> 8) & 15u')):
            L.append('  const double* __restrict__ %s = sb + %d + pg * %d + (int)(%s) * %d;'
                     % (name, self.o_tab + axis * TS, PS, sh, C + 1))
        return L

    def constants(self):
        return ['__constant__ unsigned short ib_rlane_%s[%d] = {%s};'
                % (self.tag, self.NS, ', '.join(str(c[0] | (c[1] << 4) | (c[2] << 8)) for c in self.stargets))]

    def describe(self):
        return ('Rys quadrature: %d roots, lanes own %d %s targets, %d x %d chain targets, G=%d, %d primitive quartet(s)'
                ' per product step, %d per 2D step'
                % (self.N, self.NS, self.orient, self.parts, self.nacc(), self.G, self.QPW, self.NB))

    def chunk_body(self, sync):
        """The n primitive quartets of a chunk (lane j < n holds list positions qa, qc)."""
        N, G, QPW, NB, TS, PS, C = self.N, self.G, self.QPW, self.NB, self.TS, self.PS, self.C
        o_uw, o_tab = self.o_uw, self.o_tab
        src = []
        A = src.append
        A('        if (j < n) ib_rys_setup(pd + 4 * qa, pd + 4 * (%d + qc), g, sb + j);' % PAIR_TILE)
        A('        %s;' % sync)
        A('        for (int x = j; x < n * %d; x += %d) {' % (N, G))
        A('          const int u = x / %d, rt = x - u * %d;' % (N, N))
        A('          ib_rys_root<%d>(a.rys_tab, sb[%d + u], sb[%d + u], rt, sb + %d + 2 * x);'
          % (N, 9 * CHUNK, 10 * CHUNK, o_uw))
        A('        }')
        A('        for (int b0 = 0; b0 < n; b0 += %d) {' % NB)
        A('          const int nb = min(%d, n - b0);' % NB)
        A('          %s;  // the roots are there, the last batch\'s tables are read' % sync)
        A('          for (int x = j; x < nb * %d; x += %d) {' % (3 * N, G))
        A('          const int u = x / %d, y = x - u * %d, rt = y / 3, d = y - 3 * rt;' % (3 * N, 3 * N))
        A('          const double* __restrict__ fl = sb + b0 + u;')
        A('          const double2 uw = *reinterpret_cast<const double2*>(sb + %d + 2 * ((b0 + u) * %d + rt));' % (o_uw, N))
        A('          const double B00 = uw.x * fl[%d], wt = uw.y;' % (8 * CHUNK))
        A('          const double ur0 = uw.x * fl[%d], ur1 = uw.x * fl[%d];  // u rho/zeta, u rho/eta'
          % (4 * CHUNK, 5 * CHUNK))
        A('          const double B10 = fl[%d] * (1.0 - ur0), B01 = fl[%d] * (1.0 - ur1);' % (6 * CHUNK, 7 * CHUNK))
        A('          const double ab = d == 0 ? g.AB[0] : d == 1 ? g.AB[1] : g.AB[2];')
        A('          const double cd = d == 0 ? g.CD[0] : d == 1 ? g.CD[1] : g.CD[2];')
        A('          const double pq = fl[(1 + d) * %d];' % CHUNK)
        A('          const double Cx = -fma(fl[0], ab, ur0 * pq), Dx = fma(ur1, pq, -fl[%d] * cd);' % (11 * CHUNK))
        A('          (void)B10; (void)B01; (void)Cx; (void)Dx;')
        A('          double* __restrict__ tb = sb + %d + u * %d + y * %d;' % (o_tab, PS, TS))
        src += self.chain_code()
        A('          }')
        A('          %s;' % sync)
        nops = 3 * (C + 1) + (C + 1) * (C + 2) // 2 + self.nacc()
        for h in range(self.parts):
            cond = 'own' if self.parts == 1 else 'own && part == %d' % h
            steps = NB // QPW
            if steps > 1:
                A('          if (%s)' % cond)
                A('          for (int st = 0; st < %d; ++st) {' % steps)
                A('            if (st * %d + pg >= nb) break;' % QPW)
                o = ' + st * %d' % (QPW * PS)
            else:
                A('          if (%s && pg < nb) {' % cond)
                o = ''
            A('#pragma unroll %d' % (N if N * nops <= 420 else 1))
            A('            for (int rt = 0; rt < %d; ++rt) {' % N)
            for v in 'xyz':
                A('            const double* __restrict__ t%s = pt%s%s + rt * %d;' % (v, v, o, 3 * TS))
            src += self.product_code(h)
            A('            }')
            A('          }')
        A('        }')
        return src

    def write_tables(self, nfp, tbl):
        """Accumulators -> contracted tables, one per slice and primitive quartet of a step."""
        L = []
        off = ' + pg * %d' % tbl if self.QPW > 1 else ''
        for h in range(self.parts):
            t0 = h * -(-self.NC // self.parts)
            L.append('    if (%s) {' % ('own' if self.parts == 1 else 'own && part == %d' % h))
            for k in range(len(self.part_targets(h))):
                if self.bra:
                    L.append('      sb[js * %d + %d%s] = acc[%d];' % (nfp, t0 + k, off, k))
                else:
                    L.append('      sb[%d * %d + js%s] = acc[%d];' % (t0 + k, nfp, off, k))
            L.append('    }')
        return L


class ThreadEmitter(WarpEmitter):
    """Kernel whose lanes take a primitive quartet each and run the whole
    Obara-Saika recurrence for all targets in registers (the one-thread schedule
    of eri_emitter.Emitter); the lanes' sums meet in shared memory.  For classes
    whose [e0|f0] table is small enough to be a lane's accumulators.  Bound by
    the FP64 pipe and the Boys table gathers where K is large, by latency where
    a quartet has fewer primitive quartets than lanes."""

    kind = 'thread'
    PASS = 32  # accumulators per reduction pass

    def __init__(self, la, lb, lc, ld):
        super().__init__(la, lb, lc, ld)
        self.em = Emitter(la, lb, lc, ld)
        self.vrr = self.em.emit_vrr()
        self.n = len(self.em.E) * len(self.em.F)

    def in_flight(self):
        return 2 * self.n + 20

    def nacc(self):
        return self.n

    def layout(self, tbl):
        # partial sums of a reduction pass (lane rows, odd pitch), behind the table
        self.o_red = tbl
        np = min(self.n, self.PASS)
        self.pitch = np + 1 - np % 2
        return tbl + (32 * self.pitch if self.n > 4 else 0), 1

    def constants(self):
        return []

    def describe(self):
        return 'a lane per primitive quartet, %d accumulators' % self.n

    def prologue(self):
        return []

    def chunk_body(self, sync):
        L = self.L
        src = ['        if (j < n) {',
               '        double F[%d];' % (L + 1),
               '        IbGeom q;',
               '        ib_geometry(pd + 4 * qa, pd + 4 * (%d + qc), g, q);' % PAIR_TILE,
               '        ib_boys_row<%d>(q.T, a.boys_row, F);' % L]
        if self.la + self.lb:
            src += ['        const double o2z = 0.5 * q.oz, roz = q.roz; (void)o2z; (void)roz;']
            for i, d in enumerate('xyz'):
                src.append('        const double PA%s = -q.fb * g.AB[%d], WP%s = -roz * q.PQ[%d];' % (d, i, d, i))
        if self.lc + self.ld:
            src += ['        const double o2e = 0.5 * q.oe, roe = q.roe, o2zpe = 0.5 * q.ozpe;',
                    '        (void)o2e; (void)roe; (void)o2zpe;']
            for i, d in enumerate('xyz'):
                src.append('        const double QC%s = -q.fd * g.CD[%d], WQ%s = roe * q.PQ[%d];' % (d, i, d, i))
        for m in range(L + 1):
            src.append('        const double s%d = q.pref * F[%d];' % (m, m))
        src += ['  ' + ln.replace('const R ', 'const double ').replace('(R)', '(double)').replace('(double)v', 'v')
                .replace('(double)s', 's') for ln in self.vrr]
        return src + ['        }']

    def write_tables(self, nfp, tbl):
        nf = len(self.em.F)
        at = lambda k: (k // nf) * nfp + k % nf  # noqa: E731
        L = []
        if self.n <= 4:
            L.append('    for (int o = 16; o > 0; o >>= 1) {')
            L += ['      acc[%d] += __shfl_xor_sync(0xffffffffu, acc[%d], o);' % (k, k) for k in range(self.n)]
            L.append('    }')
            L.append('    if (j == 0) {')
            L += ['      sb[%d] = acc[%d];' % (at(k), k) for k in range(self.n)]
            L.append('    }')
            return L
        L.append('    double* __restrict__ red = sb + %d;' % self.o_red)
        for k0 in range(0, self.n, self.PASS):
            m = min(self.PASS, self.n - k0)
            if k0:
                L.append('    __syncwarp();')
            L += ['    red[j * %d + %d] = acc[%d];' % (self.pitch, k, k0 + k) for k in range(m)]
            L.append('    __syncwarp();')
            L.append('    if (j < %d) {' % m)
            L.append('      double s0 = 0.0, s1 = 0.0;')
            L.append('#pragma unroll')
            L.append('      for (int v = 0; v < 32; v += 2) {')
            L.append('        s0 += red[v * %d + j];' % self.pitch)
            L.append('        s1 += red[(v + 1) * %d + j];' % self.pitch)
            L.append('      }')
            k = '%d + j' % k0 if k0 else 'j'
            L.append('      sb[(%s) / %d * %d + (%s) %% %d] = s0 + s1;' % (k, nf, nfp, k, nf))
            L.append('    }')
        return L


class RotationEmitter(WarpEmitter):
    """Rys kernel without 2D tables: three lanes per primitive quartet, ten
    primitive quartets per warp.  The targets of an s-p, p-p or s-d lane side
    fall into orbits of the cyclic axis permutation (x, xx, xy stand for all
    nine of levels 1 and 2), so lane k evaluates one representative of each
    with its axes rotated by k: the same instructions on every lane, every 2D
    integral in the lane's registers, no step between roots and products.  Bound
    by the FP64 pipe and its latency; figures at eri_emitter.ROTATED."""

    kind = 'rot'
    ORBITS = {(1, 0): ((1, 0, 0),), (1, 1): ((1, 0, 0), (2, 0, 0), (1, 1, 0)), (2, 0): ((2, 0, 0), (1, 1, 0))}
    NB = 10
    NTAB = 5      # partial tables: the second five primitive quartets add to the first five's
    chunk = 30    # three full passes

    @classmethod
    def fits(cls, la, lb, lc, ld):
        return (lc, ld) in cls.ORBITS

    def __init__(self, la, lb, lc, ld):
        super().__init__(la, lb, lc, ld)
        self.N = self.L // 2 + 1
        self.orbits = self.ORBITS[lc, ld]
        self.ctargets = comps_range(la, self.E)
        self.stargets = comps_range(lc, self.F)
        self.n = len(self.orbits) * len(self.ctargets)

    def in_flight(self):
        sx, sy = max(o[0] for o in self.orbits), max(o[1] for o in self.orbits)
        return 2 * ((self.E + 1) * (sx + sy + 3) + 12) + 16

    def nacc(self):
        return self.n

    def layout(self, tbl):
        self.o_uw = 17 * CHUNK
        self.o_tp = self.o_uw + 2 * self.N * CHUNK
        return max(self.o_tp + 2 * CHUNK, self.NTAB * tbl), self.NTAB

    def table_offset(self, orbit, c, k):
        """Offset in a contracted table of the local target (orbit, c) of lane k."""
        turn = lambda v: tuple(v[(i - k) % 3] for i in range(3))  # noqa: E731  local axis i is axis (k + i) mod 3
        nf = len(self.stargets)
        return self.ctargets.index(turn(c)) * (nf if nf % 2 else nf + 1) + self.stargets.index(turn(orbit))

    def constants(self):
        words = []
        for o in self.orbits:
            for c in self.ctargets:
                w = [self.table_offset(o, c, k) for k in range(3)]
                assert max(w) < 1024
                words.append(w[0] | (w[1] << 10) | (w[2] << 20))
        return ['__constant__ unsigned ib_rot_%s_at[%d] = {%s};' % (self.tag, self.n, ', '.join('%du' % w for w in words))]

    def describe(self):
        return 'Rys quadrature by rotated axes: %d roots, %d accumulators' % (self.N, self.n)

    def prologue(self):
        L = ['  const int pg = j / 3, rk = j % 3;  // primitive quartet of the pass, rotation',
             '  const bool own = pg < 10;']
        for i, d in enumerate('xyz'):
            L.append('  const double* __restrict__ f%s = sb + pg + ((rk + %d) %% 3) * %d;' % (d, i, 4 * CHUNK))
        return L

    def chunk_body(self, sync):
        N, C = self.N, self.E
        src = []
        A = src.append
        A('        if (j < n) ib_rot_setup(pd + 4 * qa, pd + 4 * (%d + qc), g, sb + j, sb + %d + j);' % (PAIR_TILE, self.o_tp))
        A('        %s;' % sync)
        A('        for (int x = j; x < n * %d; x += 32) {' % N)
        A('          const int u = x / %d, rt = x - u * %d;' % (N, N))
        A('          ib_rys_root<%d>(a.rys_tab, sb[%d + u], sb[%d + u], rt, sb + %d + 2 * x);'
          % (N, self.o_tp, self.o_tp + CHUNK, self.o_uw))
        A('        }')
        A('        %s;' % sync)
        A('        for (int s0 = 0; s0 < n; s0 += 10) {')
        A('          if (!(own && s0 + pg < n)) continue;')
        for d in 'xyz':
            A('          const double c%s0 = f%s[s0], c%s1 = f%s[s0 + %d], l%s0 = f%s[s0 + %d], l%s1 = f%s[s0 + %d];'
              % (d, d, d, d, CHUNK, d, d, 2 * CHUNK, d, d, 3 * CHUNK))
            A('          (void)l%s0; (void)l%s1;' % (d, d))
        A('          const double* __restrict__ fb = sb + %d + s0 + pg;' % (12 * CHUNK))
        A('          const double b0 = fb[0], b1 = fb[%d], e0 = fb[%d], e1 = fb[%d], h = fb[%d];'
          % (CHUNK, 2 * CHUNK, 3 * CHUNK, 4 * CHUNK))
        A('          (void)e0; (void)e1;')
        A('          const double2* __restrict__ uwp = reinterpret_cast<const double2*>(sb + %d) + (s0 + pg) * %d;' % (self.o_uw, N))
        A('#pragma unroll 1')
        A('          for (int rt = 0; rt < %d; ++rt) {' % N)
        A('            const double u = uwp[rt].x, wt = uwp[rt].y;')
        A('            const double CB = fma(-u, b1, b0), LB = fma(-u, e1, e0), B00 = u * h;  // chain, lane side, mixed')
        A('            (void)CB; (void)LB; (void)B00;')
        smax = (max(o[0] for o in self.orbits), max(o[1] for o in self.orbits), 0)
        val = {}
        for i, d in enumerate('xyz'):
            A('            const double C%s = fma(u, c%s1, c%s0);' % (d, d, d))
            if smax[i]:
                A('            const double L%s = fma(u, l%s1, l%s0);' % (d, d, d))

            def mul(k, a, b):  # k * a * b, with 1 dropped
                t = [x for x in ('%d.0' % k if k > 1 else None, a, b if b != '1.0' else None) if x]
                return ' * '.join(t)

            def put(c, sv, terms):
                # terms: (coefficient, factor, value) summed as FMAs, the last first
                e = mul(*terms[-1])
                for k, a, b in reversed(terms[:-1]):
                    e = 'fma(%s, %s, %s)' % (mul(k, a, '1.0'), b, e) if b != '1.0' else '%s + %s' % (mul(k, a, '1.0'), e)
                name = '%s%d_%d' % (d, c, sv)
                A('            const double %s = %s;' % (name, e))
                val[i, c, sv] = name
            val[i, 0, 0] = 'wt' if i == 2 else '1.0'
            for c in range(C):
                put(c + 1, 0, [(1, 'C' + d, val[i, c, 0])] + ([(c, 'CB', val[i, c - 1, 0])] if c else []))
            for sv in range(smax[i]):
                for c in range(C + 1):
                    put(c, sv + 1, [(1, 'L' + d, val[i, c, sv])] + ([(sv, 'LB', val[i, c, sv - 1])] if sv else []) +
                        ([(c, 'B00', val[i, c - 1, sv])] if c else []))
        yz = {}
        for o, orb in enumerate(self.orbits):
            for t, c in enumerate(self.ctargets):
                key = (c[1], orb[1], c[2])
                if key not in yz:
                    y, z = val[1, c[1], orb[1]], val[2, c[2], 0]
                    if y == '1.0':
                        yz[key] = z
                    else:
                        yz[key] = 'p%d_%d_%d' % key
                        A('            const double %s = %s * %s;' % (yz[key], y, z))
                A('            acc[%d] = fma(%s, %s, acc[%d]);'
                  % (o * len(self.ctargets) + t, val[0, c[0], orb[0]], yz[key], o * len(self.ctargets) + t))
        A('          }')
        A('        }')
        return src

    def write_tables(self, nfp, tbl):
        L = ['    double* __restrict__ mine = sb + (pg < %d ? pg : pg - %d) * %d;' % (self.NTAB, self.NTAB, tbl)]
        for half in (0, 1):
            L.append('    if (own && pg %s %d) {' % ('>=' if half else '<', self.NTAB))
            for k in range(self.n):
                L.append('      mine[(ib_rot_%s_at[%d] >> (10 * rk)) & 1023u] %s acc[%d];'
                         % (self.tag, k, '+=' if half else '=', k))
            L.append('    }')
            if not half:
                L.append('    __syncwarp();')
        return L
