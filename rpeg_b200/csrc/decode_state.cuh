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

// `chosen`, or EOS where the row's next token must be it (synthetic length control).
__device__ __forceinline__ int forced_token(const DecodeState& st, int s, int chosen) {
  const bool ends = st.active[s] && st.forced_len != nullptr && st.forced_len[s] > 0 && st.gen_count[s] + 1 >= st.forced_len[s];
  return ends ? st.eos : chosen;
}

// Record the token, retire a row that hit EOS or the cap, advance the others.
__device__ __forceinline__ void advance_row(const DecodeState& st, int s, int t, float lp) {
  if (!st.active[s]) return;
  const int g = st.gen_count[s];
  st.out_tok[static_cast<size_t>(s) * st.max_new + g] = t;
  st.out_lp[static_cast<size_t>(s) * st.max_new + g] = lp;
  st.gen_count[s] = g + 1;
  if (t == st.eos || g + 1 >= st.max_new) {
    st.active[s] = 0;
    st.seq_len[s] = 0;  // attention of a retired slot reads nothing
    atomicAdd(st.n_finished, 1);
  } else {
    st.token[s] = t;
    st.pos[s] += 1;
    st.seq_len[s] += 1;
  }
}

}  // namespace rpeg
