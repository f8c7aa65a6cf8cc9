// The state of decoding rows (see generate.cu) and what a step does to it around the choice of a token.
#pragma once

namespace rpeg {

struct DecodeState {
  const int* forced_len;
  int *token, *pos, *seq_len, *active, *gen_count, *out_tok;
  float* out_lp;
  int max_new, eos;
  int* n_finished;
  unsigned long long* step_counter;
  int* arrived;
};

// A row's state before the step, loaded at once and early: its words would be a chain of round trips behind the choice.
struct RowState {
  int active, gen_count, forced_len, pos, seq_len;
};
__device__ __forceinline__ RowState row_state(const DecodeState& st, int s) {
  return {st.active[s], st.gen_count[s], st.forced_len != nullptr ? st.forced_len[s] : 0, st.pos[s], st.seq_len[s]};
}

// `chosen`, or EOS where the row's next token must be it (synthetic length control).
__device__ __forceinline__ int forced_token(const DecodeState& st, const RowState& r, int chosen) {
  return r.active && r.forced_len > 0 && r.gen_count + 1 >= r.forced_len ? st.eos : chosen;
}

// Record the token, retire a row that hit EOS or the cap, advance the others.
__device__ __forceinline__ void advance_row(const DecodeState& st, const RowState& r, int s, int t, float lp) {
  if (!r.active) return;
  const int g = r.gen_count;
  st.out_tok[static_cast<size_t>(s) * st.max_new + g] = t;
  st.out_lp[static_cast<size_t>(s) * st.max_new + g] = lp;
  st.gen_count[s] = g + 1;
  if (t == st.eos || g + 1 >= st.max_new) {
    st.active[s] = 0;
    st.seq_len[s] = 0;  // attention of a retired slot reads nothing
    atomicAdd(st.n_finished, 1);
  } else {
    st.token[s] = t;
    st.pos[s] = r.pos + 1;
    st.seq_len[s] = r.seq_len + 1;
  }
}

}  // namespace rpeg
