// Jacobi2d chare state machine (included by jacobi2d.cu inside its
// anonymous namespace; uses JBlock, japp, jproxy and the helpers above it).
//
// State of a chare: `pass` exchanges done, `iter` sweeps done (buf[pass & 1]
// holds u_iter), `sent` = last pass whose boundary was sent, got[p] = halos
// received for the pass of parity p. A halo for pass k goes into the ghost
// zone of buf[k & 1] as soon as it is there (its sender writes it, or it is
// unpacked on arrival): pass k-1 reads only
// buf[(k-1) & 1] and writes only the interior of buf[k & 1], and a neighbour
// can be at most one pass ahead, so early halos need no stash (halo_mode 0).
// halo_mode 1 tags halos with refnum = pass instead, which parks early ones
// in the runtime's stash as the reference's refnum pattern would. Every
// chare of a problem computes the same pass lengths (pass_len), so residual
// checks fall on pass boundaries everywhere.

// Control flow is never re-entrant: pump() runs only at the top of an entry
// method; apply_decision() and tree_try_forward() report "the chare was
// parked and may continue" to their caller instead of resuming it
// themselves, so the call depth stays fixed whatever the message order.

// Thread 0: record the decision of check m.check and pass it down the tree.
// Returns 1 when the chare was parked on a decision (the block then runs
// pump()).
__device__ int apply_decision(JBlock& c, const jac::chare_desc& d, const jac::decision_msg& m) {
  if (m.check > c.decided) c.decided = m.check;
  if (m.stop && c.stop_check < 0) c.stop_check = m.check;
  c.res0 = m.res0;
  c.res_last = m.res;
  c.checks = m.check + 1;
  const int resume = c.waiting;
  c.waiting = 0;
  for (int k = 0; k < 2; k++) {
    if (d.child[k] >= 0) jproxy->invoke_single(d.child[k], EP_DECISION, &m, sizeof(m));
  }
  return resume;
}

// Thread 0: when this chare's partial and its children's are in, send the
// sum up (fixed order: own, child 0, child 1) or decide at the root. Returns
// apply_decision()'s resume flag (0 when nothing was decided). The tree's
// messages are taken and sent by thread 0 alone: as block deliveries and
// collective sends they were half of the time of small chares that check
// their residual.
__device__ int tree_try_forward(JBlock& c, const jac::chare_desc& d, int chk) {
  if (!(c.have_own && (d.child[0] < 0 || c.child_got[0]) && (d.child[1] < 0 || c.child_got[1]))) return 0;
  double t = c.own;
  if (d.child[0] >= 0) t += c.child_val[0];
  if (d.child[1] >= 0) t += c.child_val[1];
  c.have_own = 0;
  c.child_got[0] = c.child_got[1] = 0;
  if (d.parent >= 0) {
    jac::partial_msg pm;
    pm.check = chk;
    pm.slot = (d.rank - 1) % 2;
    pm.gen = c.gen;
    pm.pad = 0;
    pm.value = t;
    jproxy->invoke_single(d.parent, EP_PARTIAL, &pm, sizeof(pm));
    return 0;
  }
  const jac::prob_desc& p = c.prob;
  const double nrm = sqrt(t);
  jac::decision_msg dm;
  dm.check = chk;
  dm.gen = c.gen;
  dm.pad = 0;
  dm.res0 = (chk == 0) ? nrm : c.res0;
  dm.res = nrm;
  dm.stop = (p.tol > 0.0) && (dm.res0 == 0.0 || nrm <= p.tol * dm.res0) ? 1 : 0;
  return apply_decision(c, d, dm);
}

// All threads: one pass buf[pass&1] -> buf[(pass+1)&1], then the residual
// tree when the pass starts at a check.
template <typename T>
__device__ void advance(JBlock& c, const jac::chare_desc& d) {
  const jac::prob_desc& p = c.prob;
  int K = p.check_every;
  // read before thread 0 advances the chare below
  const bool resid = K > 0 && (c.iter % K == 0);
  const int chk = K > 0 ? c.iter / K : 0;
  const int L = pass_len(d, p, c.iter);
  double part = sweep_block<T>(d, c.cur, resid, L);
  if (threadIdx.x == 0) {
    c.got[c.pass & 1] = 0;
    c.gotx[c.pass & 1] = 0;
    c.cur ^= 1;
    c.pass++;
    c.iter += L;
    if (resid) {
      c.own = part;
      c.have_own = 1;
      // A decision taken here (at the tree root) cannot find this chare
      // parked: it is sweeping. pump()'s loop re-examines the state anyway.
      (void)tree_try_forward(c, d, chk);
    }
  }
  __syncthreads();
}

// All threads: drive the chare as far as it can go without new messages:
// decide (stop / park on a residual decision / continue), send the boundary
// of u_iter once, and sweep whenever all halos of the current sweep are in.
template <typename T>
__device__ void pump(JBlock& c, const jac::chare_desc& d) {
  const jac::prob_desc& p = c.prob;
  __shared__ int s_act;
  enum { IDLE = 0, SEND = 1, FIN = 2, SWEEP = 3, SELF = 4, SEND_Y = 5 };
  // lattice updates a chare without neighbours may run in one entry method
  // (a message round trip costs about as much as 20 K of them)
  long long self_budget = 1ll << 18;
  while (true) {
    if (threadIdx.x == 0) {
      int act = IDLE;
      int K = p.check_every;
      (void)CHARM_VERIFY(c.cur == (c.pass & 1) && c.got[0] <= c.nbr_count && c.got[1] <= c.nbr_count,
                   CHARMING_ERR_APP, 7000 + c.pass, c.i);
      if (c.done || c.waiting) {
        act = IDLE;
      } else if (c.sent < c.pass) {
        if (c.iter >= p.max_sweeps) {
          // finish only after the decision of the last residual check: the
          // result reports that check's norm, and no message of the problem
          // is left in flight (a serving worker can take the next request)
          if (K > 0 && p.max_sweeps > 0 && c.decided < (p.max_sweeps - 1) / K) {
            c.waiting = 1;
            act = IDLE;
          } else {
            act = FIN;
          }
        } else if (K > 0 && c.iter >= K && c.iter % K == 0 && c.decided < c.iter / K - 1) {
          c.waiting = 1;
          act = IDLE;
        } else if (K > 0 && c.iter >= K && c.iter % K == 0 && c.stop_check >= 0 &&
                   c.stop_check <= c.iter / K - 1) {
          act = FIN;
        } else {
          act = c.nbr_count > 0 ? SEND : SELF;
          c.sent = c.pass;
          if (act == SEND && japp::halo_mode() == 1) jproxy->set_refnum(c.i, c.pass);
        }
      } else if (d.ext > 0 && c.sent_y < c.pass && c.gotx[c.pass & 1] == c.nbx) {
        // two-phase: the left/right ghost columns of this pass are in, so
        // the top/bottom halos can carry the corners
        act = SEND_Y;
        c.sent_y = c.pass;
      } else if (c.nbr_count > 0 && c.got[c.pass & 1] == c.nbr_count && (d.ext == 0 || c.sent_y == c.pass)) {
        act = SWEEP;
      }
      s_act = act;
    }
    __syncthreads();
    int act = s_act;
    __syncthreads();
    if (act == IDLE) return;
    if (act == FIN) {
      finish(c, d);
      return;
    }
    if (act == SEND) {
      send_halos<T>(c, d, d.ext > 0 ? 1 : 0);
    } else if (act == SEND_Y) {
      send_halos<T>(c, d, 2);
    } else if (act == SELF) {
      // no neighbours: passes back to back up to a work budget, then one
      // message to itself, so other chares of the PE run in between
      if (self_budget > 0) {
        self_budget -= (long long)d.w * d.h * pass_len(d, p, c.iter);
        advance<T>(c, d);
        continue;
      }
      int it = c.pass;
      jproxy->invoke(c.i, EP_CONT, &it, sizeof(int));
      return;
    } else {
      advance<T>(c, d);
    }
  }
}

template <typename T>
__device__ void em_start_t(JBlock& c, void* arg) {
  if (japp::serving()) {
    // the start of a request travels down the residual tree
    const jac::start_msg m = *reinterpret_cast<const jac::start_msg*>(arg);
    if (!ensure_gen<T>(c, m.gen)) return;
    const jac::chare_desc& d = c.desc;
    for (int k = 0; k < 2; k++) {
      jac::start_msg f = m;
      if (d.child[k] >= 0) jproxy->invoke(d.child[k], EP_START, &f, sizeof(f));
    }
    pump<T>(c, d);
    return;
  }
  const jac::chare_desc& d = c.desc;
  if (threadIdx.x == 0) {
    count_nbrs(c, d);
    c.started = 1;
  }
  __syncthreads();
  pump<T>(c, d);
}

template <typename T>
__device__ void em_halo_t(JBlock& c, void* arg) {
  const jac::halo_hdr* hh = reinterpret_cast<const jac::halo_hdr*>(arg);
  if (!ensure_gen<T>(c, hh->gen)) return;
  if (c.done) return;
  const unsigned long long t_em = threadIdx.x == 0 ? pe_clock() : 0;
  const jac::chare_desc& d = c.desc;
  // checked build: direction, length and sweep of the halo are consistent
  if (!CHARM_VERIFY(hh->dir >= 0 && hh->dir < jac::N_DIRS && d.nbr[hh->dir] >= 0, CHARMING_ERR_APP,
                    1000 + hh->dir, c.i) ||
      !CHARM_VERIFY(hh->len == jac::halo_ghost(hh->dir, d).nr * jac::halo_ghost(hh->dir, d).nc,
                    CHARMING_ERR_APP, 2000 + hh->dir, hh->len) ||
      !CHARM_VERIFY(hh->pass == c.pass || hh->pass == c.pass + 1, CHARMING_ERR_APP,
                    3000 + (hh->pass - c.pass), c.i))
    return;
  unpack_halo<T>(c, d, arg);
  if (threadIdx.x == 0) {
    c.got[hh->pass & 1]++;
    if (hh->dir == jac::LEFT || hh->dir == jac::RIGHT) c.gotx[hh->pass & 1]++;
    (void)CHARM_VERIFY(c.got[hh->pass & 1] <= jac::N_DIRS, CHARMING_ERR_APP, 4000 + c.got[hh->pass & 1], c.i);
  }
  __syncthreads();
  if (threadIdx.x == 0) add_pe_cyc(2, pe_clock() - t_em);
  if (c.started) pump<T>(c, d);  // a halo may overtake the start message
}

template <typename T>
__device__ void em_cont_t(JBlock& c) {
  if (c.done) return;
  const jac::chare_desc& d = c.desc;
  advance<T>(c, d);
  pump<T>(c, d);
}

// ---- inline entry methods (thread 0) ----------------------------------------
// A message of a newer request than the worker's (serving) goes to the block,
// which sets the request up first; one of an older request is dropped.
__device__ __forceinline__ int stale(const JBlock& c, unsigned gen, int fresh_ep) {
  if (!japp::serving() || gen == c.gen) return 0;
  return gen > c.gen ? fresh_ep : -1;
}

// A neighbour's halo of hh->pass lies in the ghost zone: count it; the block
// runs when the chare can go on (the conditions of pump()).
__device__ int in_note(JBlock& c, void* arg) {
  const jac::halo_hdr* hh = reinterpret_cast<const jac::halo_hdr*>(arg);
  const int dir = hh->dir, pass = hh->pass;
  if (const int s = stale(c, hh->gen, EP_FRESH_NOTE)) return s;
  if (c.done) return -1;
  if (!CHARM_VERIFY(dir >= 0 && dir < 4 && c.desc.nbr[dir] >= 0, CHARMING_ERR_APP, 1000 + dir, c.i) ||
      !CHARM_VERIFY(pass == c.pass || pass == c.pass + 1, CHARMING_ERR_APP, 3000 + (pass - c.pass), c.i))
    return -1;
  c.got[pass & 1]++;
  if (dir == jac::LEFT || dir == jac::RIGHT) c.gotx[pass & 1]++;
  if (!c.started || c.waiting || c.sent < c.pass) return -1;  // (the start pumps; so does a decision)
  if (c.desc.ext > 0 && c.sent_y < c.pass) return c.gotx[c.pass & 1] == c.nbx ? EP_PUMP : -1;
  return c.got[c.pass & 1] == c.nbr_count ? EP_PUMP : -1;
}

__device__ int in_partial(JBlock& c, void* arg) {
  const jac::partial_msg m = *reinterpret_cast<const jac::partial_msg*>(arg);
  if (const int s = stale(c, m.gen, EP_FRESH_PARTIAL)) return s;
  if (c.done) return -1;
  const jac::chare_desc& d = c.desc;
  if (!CHARM_VERIFY(m.slot == 0 || m.slot == 1, CHARMING_ERR_APP, 5000 + m.slot, c.i) ||
      !CHARM_VERIFY(d.child[m.slot] >= 0 && !c.child_got[m.slot], CHARMING_ERR_APP, 6000 + m.slot, c.i))
    return -1;
  c.child_val[m.slot] = m.value;
  c.child_got[m.slot] = 1;
  return tree_try_forward(c, d, m.check) ? EP_PUMP : -1;
}

__device__ int in_decision(JBlock& c, void* arg) {
  const jac::decision_msg m = *reinterpret_cast<const jac::decision_msg*>(arg);
  if (const int s = stale(c, m.gen, EP_FRESH_DECISION)) return s;
  if (c.done) return -1;
  return apply_decision(c, c.desc, m) ? EP_PUMP : -1;
}

// The request generation a message of inline entry method In carries.
template <int In(JBlock&, void*)>
__device__ unsigned msg_gen(const void* arg);
template <>
__device__ unsigned msg_gen<in_note>(const void* arg) { return reinterpret_cast<const jac::halo_hdr*>(arg)->gen; }
template <>
__device__ unsigned msg_gen<in_partial>(const void* arg) { return reinterpret_cast<const jac::partial_msg*>(arg)->gen; }
template <>
__device__ unsigned msg_gen<in_decision>(const void* arg) { return reinterpret_cast<const jac::decision_msg*>(arg)->gen; }
