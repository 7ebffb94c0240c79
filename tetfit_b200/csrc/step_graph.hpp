// Capture of launched steps into an executable graph.  A capture that the
// runtime refuses leaves the stream as it was and no graph: the caller then
// launches its steps one by one (same kernels, same results).  The runtime's
// calls come in through Api (cuda_util.hpp: CudaGraphs).
#pragma once

namespace tf {

template <typename Api, typename Launch>
typename Api::Exec capture_steps(typename Api::Stream stream, Launch launch) {
  typename Api::Exec exec = nullptr;
  if (!Api::begin(stream)) {
    Api::clear_error();
    return nullptr;
  }
  bool ok = true;
  try {
    launch();
  } catch (...) {
    ok = false;  // a launch the capture refused; the capture is ended all the same
  }
  typename Api::Graph graph = nullptr;
  ok = Api::end(stream, &graph) && ok;
  if (ok && !Api::instantiate(&exec, graph)) exec = nullptr;
  if (graph) Api::destroy(graph);
  if (!exec) Api::clear_error();
  return exec;
}

}  // namespace tf
